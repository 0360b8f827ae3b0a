// Results to host memory (see readback.hpp).  Host code over the CUDA runtime only.
#include "readback.hpp"

#include <sys/mman.h>
#include <unistd.h>

#include <algorithm>
#include <cstdint>
#include <cstring>
#include <exception>
#include <thread>
#include <vector>

#include "cuda_check.hpp"

namespace olfb200 {

HostReadback::~HostReadback() { release(); }

void HostReadback::release() {
    for (cudaEvent_t& e : ready) {
        if (e) cudaEventDestroy(e);
        e = nullptr;
    }
    if (ring) cudaFreeHost(ring);
    ring = nullptr;
}

// The ring and its events, all or none of them; after a failure the direct copies stay.
void HostReadback::makeRing() {
    bool ok = cudaMallocHost(reinterpret_cast<void**>(&ring), SLOTS * CHUNK) == cudaSuccess;
    if (!ok) ring = nullptr;
    for (int k = 0; ok && k < SLOTS; k++) {
        ok = cudaEventCreateWithFlags(&ready[k], cudaEventDisableTiming) == cudaSuccess;
        if (!ok) ready[k] = nullptr;
    }
    if (!ok) release();
    failed = !ok;
}

// At least half of the array's pages (fewer than LARGE bytes) have memory behind them already.
bool HostReadback::inMemory(const void* p, size_t bytes) {
    const uintptr_t page = static_cast<uintptr_t>(sysconf(_SC_PAGESIZE));
    const uintptr_t from = reinterpret_cast<uintptr_t>(p) / page * page;
    const size_t pages = (reinterpret_cast<uintptr_t>(p) + bytes - from + page - 1) / page;
    unsigned char there[LARGE / 4096 + 2];
    if (pages > sizeof(there) || mincore(reinterpret_cast<void*>(from), pages * page, there) != 0) return true;
    size_t n = 0;
    for (size_t k = 0; k < pages; k++) n += there[k] & 1;
    return 2 * n >= pages;
}

bool HostReadback::copy(int device, void* dst, const void* src, size_t bytes, cudaStream_t st) {
    const ErrorMark mark;      // the caller's launches before the copy are checked after it
    cudaPointerAttributes at{};
    const bool known = cudaPointerGetAttributes(&at, dst) == cudaSuccess;
    if (!known) mark.drop();
    const bool pageable = known && at.type == cudaMemoryTypeUnregistered;
    const bool worth = pageable && bytes >= 2 * CHUNK && (bytes >= LARGE || !inMemory(dst, bytes));
    if (worth) due += bytes;
    if (worth && !ring && !failed && due >= EARNED) {
        makeRing();
        if (failed) mark.drop();
    }
    if (!worth || !ring) {
        OLF_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, st));
        return true;
    }
    const size_t chunks = (bytes + CHUNK - 1) / CHUNK;
    cudaError_t err[SLOTS] = {};
    auto work = [&](int slot, int slots) {
        err[slot] = cudaSetDevice(device);
        for (size_t c = slot; c < chunks && err[slot] == cudaSuccess; c += slots) {
            const size_t at0 = c * CHUNK, len = std::min(CHUNK, bytes - at0);
            unsigned char* pin = ring + static_cast<size_t>(slot) * CHUNK;
            cudaError_t e = cudaMemcpyAsync(pin, static_cast<const unsigned char*>(src) + at0, len, cudaMemcpyDeviceToHost, st);
            if (e == cudaSuccess) e = cudaEventRecord(ready[slot], st);
            if (e == cudaSuccess) e = cudaEventSynchronize(ready[slot]);
            if (e == cudaSuccess) std::memcpy(static_cast<unsigned char*>(dst) + at0, pin, len);
            err[slot] = e;
        }
    };
    const int slots = static_cast<int>(std::min<size_t>(chunks, std::min(SLOTS, std::max(1, static_cast<int>(std::thread::hardware_concurrency()) / 2))));
    std::vector<std::thread> threads;
    int mine = 0;     // slots whose thread could not be started run here
    try {
        threads.reserve(slots);
        for (int k = 1; k < slots; k++) threads.emplace_back(work, k, slots);
    } catch (const std::exception&) {      // std::system_error, std::bad_alloc: the threads that run are joined below
        mine = static_cast<int>(threads.size()) + 1;
    }
    work(0, slots);
    for (int k = mine; mine > 0 && k < slots; k++) work(k, slots);
    for (std::thread& t : threads) t.join();
    for (int k = 0; k < slots; k++) OLF_CUDA(err[k]);
    return false;
}

}  // namespace olfb200
