// hostcopy.cuh -- large copies between the device and ordinary (pageable) host memory.
#pragma once
#include <cuda_runtime.h>
#include <cstddef>

namespace wg {

// The page-locked slots of one context's large copies (HC_LANES x 2 x HC_CHUNK bytes),
// made at the first of them and kept until host_copy_free.
constexpr int HC_LANES = 8;              // host threads of a copy, at most
constexpr size_t HC_CHUNK = 512 << 10;
constexpr size_t HC_MIN = 4 << 20;       // smaller copies are left to cudaMemcpyAsync
struct HostCopy {
    char* pin = nullptr;
    cudaStream_t st[HC_LANES] = {};
    cudaEvent_t ev[HC_LANES][2] = {};
    bool off = false;                    // the slots could not be made: plain copies from then on
};

// cudaMemcpyAsync(dst, src, bytes, kind, s) for kind host to device or device to host; a
// large copy of pageable memory has ended, after all earlier work of s, when it returns.
cudaError_t host_copy(HostCopy* h, int device, void* dst, const void* src, size_t bytes, cudaMemcpyKind kind,
                      cudaStream_t s);
void host_copy_free(HostCopy* h);

}  // namespace wg
