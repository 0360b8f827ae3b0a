// HostReadback (csrc/readback.cpp) over a stand-in for the CUDA runtime in host memory: which errors it leaves behind, what it
// holds after a failure, and the bytes it brings.  Usage: readback_host <case>; prints "ok" or what went wrong.
#include <dlfcn.h>
#include <pthread.h>
#include <sys/mman.h>

#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <new>
#include <string>
#include <vector>

#include "../../olf-gpu_b200/csrc/readback.hpp"

namespace {
thread_local cudaError_t last = cudaSuccess;       // the runtime's last error is per host thread
std::atomic<int> pinned{0}, pinCalls{0}, eventsMade{0}, eventsGone{0}, directCopies{0}, ringCopies{0};
bool failQuery = false, failPin = false;
int failEventAt = -1, failThreadAt = -1, failNewAt = -1;
std::atomic<int> threadCalls{0}, newCalls{0};
std::mutex copies;
unsigned char* ringLo = nullptr;
size_t ringBytes = 0;
void* pinnedDst = nullptr;

cudaError_t fail(cudaError_t e) { return last = e; }
}  // namespace

extern "C" {
cudaError_t cudaPeekAtLastError() { return last; }
cudaError_t cudaGetLastError() {
    const cudaError_t e = last;
    last = cudaSuccess;
    return e;
}
const char* cudaGetErrorString(cudaError_t) { return "stand-in error"; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* at, const void* p) {
    if (failQuery) return fail(cudaErrorInvalidValue);
    at->type = p == pinnedDst ? cudaMemoryTypeHost : cudaMemoryTypeUnregistered;
    return cudaSuccess;
}
cudaError_t cudaMallocHost(void** p, size_t n) {
    pinCalls++;
    if (failPin) return fail(cudaErrorMemoryAllocation);
    *p = std::malloc(n);
    ringLo = static_cast<unsigned char*>(*p);
    ringBytes = n;
    pinned++;
    return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p) {
    std::free(p);
    pinned--;
    return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
    if (failEventAt >= 0 && eventsMade == failEventAt) return fail(cudaErrorMemoryAllocation);
    *e = reinterpret_cast<cudaEvent_t>(static_cast<size_t>(++eventsMade));
    return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t) {
    eventsGone++;
    return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t) { return e ? cudaSuccess : fail(cudaErrorInvalidResourceHandle); }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* dst, const void* src, size_t n, cudaMemcpyKind, cudaStream_t) {
    std::lock_guard<std::mutex> lock(copies);
    const bool ring = static_cast<unsigned char*>(dst) >= ringLo && static_cast<unsigned char*>(dst) < ringLo + ringBytes;
    (ring ? ringCopies : directCopies)++;
    std::memcpy(dst, src, n);
    return cudaSuccess;
}
int pthread_create(pthread_t* t, const pthread_attr_t* a, void* (*f)(void*), void* x) {
    if (failThreadAt >= 0 && threadCalls++ >= failThreadAt) return EAGAIN;
    using Create = int (*)(pthread_t*, const pthread_attr_t*, void* (*)(void*), void*);
    return reinterpret_cast<Create>(dlsym(RTLD_NEXT, "pthread_create"))(t, a, f, x);
}
}

void* operator new(size_t n) {
    if (failNewAt >= 0 && newCalls++ == failNewAt) throw std::bad_alloc();
    void* p = std::malloc(n ? n : 1);
    if (!p) throw std::bad_alloc();
    return p;
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, size_t) noexcept { std::free(p); }

namespace {
constexpr size_t MIB = size_t(1) << 20;
const char* wrong = nullptr;
void expect(bool ok, const char* what) {
    if (!ok && !wrong) wrong = what;
}

// One copy of n bytes, to a fresh array or to one whose pages are in memory; its bytes are compared and whether it threw
// returned.
enum Kind { FRESH, USED, PINNED };
bool copyOnce(olfb200::HostReadback& r, size_t n, Kind kind = FRESH) {
    std::vector<unsigned char> src(n);
    for (size_t i = 0; i < n; i++) src[i] = static_cast<unsigned char>(i * 2654435761u >> 24);
    unsigned char* dst = static_cast<unsigned char*>(
        mmap(nullptr, n, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0));
    if (kind != FRESH) std::memset(dst, 0, n);
    pinnedDst = kind == PINNED ? dst : nullptr;
    bool threw = false;
    try {
        r.copy(0, dst, src.data(), n, nullptr);
    } catch (const std::exception&) {
        threw = true;
    }
    if (!threw) expect(std::memcmp(src.data(), dst, n) == 0, "bytes differ");
    munmap(dst, n);
    return threw;
}

// After a launch that failed before the copy, the thread still has an error to report, whatever the copy itself meets.
void pendingError() {
    for (int variant = 0; variant < 3; variant++) {
        failQuery = variant == 1;
        failPin = variant == 2;
        olfb200::HostReadback r;
        for (const size_t n : {MIB / 4, 3 * MIB, 20 * MIB}) {
            for (const Kind kind : {FRESH, USED, PINNED}) {
                last = cudaErrorInvalidConfiguration;
                expect(!copyOnce(r, n, kind), "copy threw");
                expect(last != cudaSuccess, "a pending launch error was cleared");
            }
        }
    }
}

// What the copy's own failed calls set does not outlive it.
void ownError() {
    for (const bool query : {false, true}) {
        failQuery = query;
        failPin = !query;
        olfb200::HostReadback r;
        for (int k = 0; k < 3; k++) expect(!copyOnce(r, 20 * MIB), "copy threw");
        expect(last == cudaSuccess, "the copy left an error behind");
    }
}

// A ring that cannot be pinned: copied directly, tried once, and no event held or lost.
void pinFails() {
    failPin = true;
    {
        olfb200::HostReadback r;
        for (int k = 0; k < 4; k++) expect(!copyOnce(r, 20 * MIB), "copy threw");
        expect(directCopies == 4, "not copied directly");
        expect(pinCalls == 1, "pinned again after a failure");
    }
    expect(eventsMade == eventsGone, "events lost");
}

// An event that cannot be made: the ring and the events made before it are given back, copied directly.
void eventFails() {
    failEventAt = 3;
    {
        olfb200::HostReadback r;
        for (int k = 0; k < 3; k++) expect(!copyOnce(r, 20 * MIB), "copy threw");
        expect(directCopies == 3, "not copied directly");
    }
    expect(pinned == 0, "ring lost");
    expect(eventsMade == eventsGone, "events lost");
    expect(last == cudaSuccess, "the copy left an error behind");
}

// Threads that cannot be started (by the system, or for want of memory): their chunks are copied by the others.
void threadsFail() {
    for (int at = 0; at < 8; at++) {
        olfb200::HostReadback r;
        failThreadAt = -1;
        expect(!copyOnce(r, 20 * MIB), "copy threw");
        threadCalls = 0;
        failThreadAt = at;
        expect(!copyOnce(r, 20 * MIB + 5), "copy threw");
    }
}
void memoryFails() {
    for (int at = 0; at < 12; at++) {
        olfb200::HostReadback r;
        std::vector<unsigned char> src(20 * MIB, 7), dst(20 * MIB, 0);
        pinnedDst = nullptr;
        r.copy(0, dst.data(), src.data(), src.size(), nullptr);
        std::memset(dst.data(), 0, dst.size());
        newCalls = 0;
        failNewAt = at;
        try {
            r.copy(0, dst.data(), src.data(), src.size(), nullptr);
            failNewAt = -1;
            expect(src == dst, "bytes differ");
        } catch (const std::exception&) {
            failNewAt = -1;      // before any thread ran: an error is as good
        }
    }
}

// Sizes around the thresholds, the chunks and the slots.
void sizes() {
    olfb200::HostReadback r;
    for (const size_t n : {size_t(1), MIB / 2, MIB - 1, MIB, MIB + 1, 4 * MIB - 8, 4 * MIB, 4 * MIB + 8, 17 * MIB + 3,
                           32 * MIB - 1, 32 * MIB, 33 * MIB + 5})
        for (const Kind kind : {FRESH, USED, PINNED, FRESH}) expect(!copyOnce(r, n, kind), "copy threw");
    expect(ringCopies > 0, "the ring never ran");
}

// Which way a copy takes: arrays in memory directly up to 32 MiB, fresh ones through the ring once it has been earned.
void ways() {
    olfb200::HostReadback r;
    auto direct = [&](size_t n, Kind kind) {
        const int before = directCopies;
        expect(!copyOnce(r, n, kind), "copy threw");
        return directCopies == before + 1;
    };
    for (int k = 0; k < 20; k++) expect(direct(4 * MIB, USED), "an array in memory went through the ring");
    expect(pinCalls == 0, "the ring was pinned for arrays in memory");
    for (int k = 0; k < 3; k++) expect(direct(4 * MIB, FRESH), "the ring was pinned before it was earned");
    expect(!direct(4 * MIB, FRESH), "a fresh array was copied directly");
    expect(direct(MIB - 1, FRESH) && direct(4 * MIB, USED) && direct(20 * MIB, PINNED), "a copy went through the ring");
    expect(direct(32 * MIB - 1, USED), "an array in memory went through the ring");
    expect(!direct(32 * MIB, USED), "a large copy was made directly");
    expect(pinCalls == 1, "more than one ring");
}
}  // namespace

int main(int argc, char** argv) {
    const std::string c = argc > 1 ? argv[1] : "";
    if (c == "pending") pendingError();
    else if (c == "own") ownError();
    else if (c == "pin") pinFails();
    else if (c == "event") eventFails();
    else if (c == "threads") threadsFail();
    else if (c == "memory") memoryFails();
    else if (c == "sizes") sizes();
    else if (c == "ways") ways();
    else wrong = "unknown case";
    std::puts(wrong ? wrong : "ok");
    return wrong ? 1 : 0;
}
