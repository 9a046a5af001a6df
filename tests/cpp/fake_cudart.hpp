// fake_cudart.hpp — the CUDA runtime entry points that the library's host code
// calls, on host memory and without a device: allocations are malloc, copies
// are memcpy, streams and events are empty, and a launch runs nothing but a
// hook.  A test links the library's own objects against it to see what their
// host side does: which launches it makes and with which sizes, and what
// becomes of a launch that the runtime refuses.
#pragma once

#include <cuda_runtime.h>

#include <functional>
#include <map>
#include <set>
#include <string>

namespace fake {

struct Launch {
    std::string kernel;  // mangled name
    dim3 grid, block;
    size_t smem = 0;
    void** args = nullptr;
};
inline std::map<const void*, std::string>& names() {  // filled before main
    static std::map<const void*, std::string> n;
    return n;
}
// per kernel: every value given to its dynamic shared memory limit
inline std::map<std::string, std::set<int>> smem_limit;
inline std::function<cudaError_t(const Launch&)> on_launch;
inline std::function<cudaError_t(const std::string&)> on_attribute;
inline cudaError_t last_error = cudaSuccess;

}  // namespace fake

