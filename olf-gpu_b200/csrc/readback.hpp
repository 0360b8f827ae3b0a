// Results to host memory.
#pragma once

#include <cuda_runtime_api.h>

#include <cstddef>

namespace olfb200 {

// Brings large results to pageable host memory through a small pinned ring, several threads copying out of it (and taking
// the page faults of a fresh array) while the next chunks cross the bus.  Pinned or small destinations are copied directly.
// 74 MB of results to a fresh array: 5 ms, against 26 ms for one pageable copy; 4.8 MB: the pageable copy takes 3 ms.
class HostReadback {
public:
    HostReadback() = default;
    HostReadback(const HostReadback&) = delete;
    HostReadback& operator=(const HostReadback&) = delete;
    ~HostReadback();
    // Stream-ordered after what st holds; true: enqueued on st (the caller synchronises), false: the copy is complete.
    bool copy(int device, void* dst, const void* src, size_t bytes, cudaStream_t st);

private:
    static constexpr size_t CHUNK = size_t(512) << 10;   // (a 4 MiB ring: pinning 16 MiB cost a new context 5 ms)
    static constexpr int SLOTS = 8;
    unsigned char* ring = nullptr;      // pinned, SLOTS chunks, made on the first large or the second smaller copy
    bool seen = false, failed = false;  // failed: the ring could not be made, and is not tried again
    cudaEvent_t ready[SLOTS] = {};
    void makeRing();
    void release();
};

}  // namespace olfb200
