// Results to host memory.
#pragma once

#include <cuda_runtime_api.h>

#include <cstddef>

namespace olfb200 {

// Brings large results to pageable host memory through a small pinned ring, several threads copying out of it (and taking
// the page faults of a fresh array) while the next chunks cross the bus.
//
// What it is worth depends on the array.  Fresh pages cost more than the copy, and the threads share them; in an array that
// is in memory already the threads' start is all that is added, until the copy itself is long enough to share.  Whole solves
// on 9,241 buses, direct copy / ring, results kept (fresh arrays): 2.4 MiB 3.6 / 3.0 ms, 9.2 MiB 7.4 / 5.9, 18 MiB 10.4 /
// 6.9; results dropped (the allocator hands out the same pages): 2.4 MiB 2.75 / 3.2 ms, 9.2 MiB 5.9 / 6.8, 18 MiB 7.6 / 7.9,
// 37 MiB (fresh again: the allocator returns arrays of 32 MiB to the system) 16.3 / 10.5.  So: fresh arrays from two chunks on
// (1.1 MiB 2.62 / 2.51 ms), others from LARGE on; pinned memory is copied directly.  Pinning the ring costs 3 to 8 ms once: it
// is made when the copies it is for have added up to EARNED, about what it saves on them.
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
    static constexpr size_t LARGE = size_t(32) << 20, EARNED = size_t(16) << 20;
    unsigned char* ring = nullptr;      // pinned, SLOTS chunks
    size_t due = 0;                     // bytes of the copies that the ring is for, so far
    bool failed = false;                // the ring could not be made, and is not tried again
    cudaEvent_t ready[SLOTS] = {};
    static bool inMemory(const void* p, size_t bytes);
    void makeRing();
    void release();
};

}  // namespace olfb200
