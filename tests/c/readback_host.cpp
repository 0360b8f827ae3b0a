// HostReadback (csrc/readback.cpp) over a stand-in for the CUDA runtime in host memory: which errors it leaves behind
// and the bytes it brings.  Usage: readback_host <case>; prints "ok" or what went wrong.
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <string>
#include <vector>

#include "../../olf-gpu_b200/csrc/readback.hpp"

namespace {
thread_local cudaError_t last = cudaSuccess;       // the runtime's last error is per host thread
std::atomic<int> eventsMade{0}, directCopies{0}, ringCopies{0};
bool failQuery = false, failPin = false;
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
    if (failPin) return fail(cudaErrorMemoryAllocation);
    *p = std::malloc(n);
    ringLo = static_cast<unsigned char*>(*p);
    ringBytes = n;
    return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p) {
    std::free(p);
    return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
    *e = reinterpret_cast<cudaEvent_t>(static_cast<size_t>(++eventsMade));
    return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t) { return e ? cudaSuccess : fail(cudaErrorInvalidResourceHandle); }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* dst, const void* src, size_t n, cudaMemcpyKind, cudaStream_t) {
    std::lock_guard<std::mutex> lock(copies);
    const bool ring = static_cast<unsigned char*>(dst) >= ringLo && static_cast<unsigned char*>(dst) < ringLo + ringBytes;
    (ring ? ringCopies : directCopies)++;
    std::memcpy(dst, src, n);
    return cudaSuccess;
}
}

namespace {
constexpr size_t MIB = size_t(1) << 20;
const char* wrong = nullptr;
void expect(bool ok, const char* what) {
    if (!ok && !wrong) wrong = what;
}

// One copy of n bytes; its bytes are compared and whether it threw returned.
bool copyOnce(olfb200::HostReadback& r, size_t n, bool toPinned = false) {
    std::vector<unsigned char> src(n), dst(n, 0);
    for (size_t i = 0; i < n; i++) src[i] = static_cast<unsigned char>(i * 2654435761u >> 24);
    pinnedDst = toPinned ? dst.data() : nullptr;
    bool threw = false;
    try {
        r.copy(0, dst.data(), src.data(), n, nullptr);
    } catch (const std::exception&) {
        threw = true;
    }
    if (!threw) expect(std::memcmp(src.data(), dst.data(), n) == 0, "bytes differ");
    return threw;
}

// After a launch that failed before the copy, the thread still has an error to report, whatever the copy itself meets.
void pendingError() {
    for (int variant = 0; variant < 3; variant++) {
        failQuery = variant == 1;
        failPin = variant == 2;
        olfb200::HostReadback r;
        for (const size_t n : {MIB / 4, 3 * MIB, 20 * MIB}) {
            for (const bool toPinned : {false, true}) {
                last = cudaErrorInvalidConfiguration;
                expect(!copyOnce(r, n, toPinned), "copy threw");
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

// Sizes around the threshold, the chunks and the slots.
void sizes() {
    olfb200::HostReadback r;
    for (const size_t n : {size_t(1), MIB / 2, MIB - 1, MIB, MIB + 1, 4 * MIB - 8, 4 * MIB, 4 * MIB + 8, 17 * MIB + 3})
        for (int k = 0; k < 2; k++) expect(!copyOnce(r, n), "copy threw");
    expect(ringCopies > 0, "the ring never ran");
}
}  // namespace

int main(int argc, char** argv) {
    const std::string c = argc > 1 ? argv[1] : "";
    if (c == "pending") pendingError();
    else if (c == "own") ownError();
    else if (c == "sizes") sizes();
    else wrong = "unknown case";
    std::puts(wrong ? wrong : "ok");
    return wrong ? 1 : 0;
}
