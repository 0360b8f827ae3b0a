// CUDA status checks of the host code.
#pragma once

#include <cuda_runtime_api.h>

#include <stdexcept>
#include <string>

#define OLF_CUDA(call)                                                                                              \
    do {                                                                                                            \
        cudaError_t err_ = (call);                                                                                  \
        if (err_ != cudaSuccess) {                                                                                  \
            throw std::runtime_error(std::string("CUDA error ") + cudaGetErrorString(err_) + " at " __FILE__ ":" + \
                                     std::to_string(__LINE__));                                                     \
        }                                                                                                           \
    } while (0)

namespace olfb200 {

// For calls that may fail without harm: drop() forgets what they left as the thread's last error, but not an error that was
// there before them (a launch that failed, which the solve still has to report).
struct ErrorMark {
    const cudaError_t before = cudaPeekAtLastError();
    void drop() const {
        if (before == cudaSuccess) cudaGetLastError();
    }
};

}  // namespace olfb200
