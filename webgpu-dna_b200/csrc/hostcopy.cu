// hostcopy.cu -- large copies between the device and ordinary (pageable) host memory.
//
// What bounds such a copy is the host: cudaMemcpyAsync moves pageable memory through a
// staging buffer with one thread, which also takes the first-touch page faults of a
// fresh buffer.  Here up to HC_LANES threads each move a contiguous part of it through
// two page-locked slots of their own, so that the DMA of one chunk runs while the
// thread copies the other.  Memory that is page-locked already is left to the DMA
// alone, and so is what is smaller than HC_MIN, where the threads' start costs what it gives.
// Measured (ms, cudaMemcpyAsync and this, 16 host cores): to a fresh buffer 85 MB 18.8 and
// 3.5, 34 MB 7.1 and 1.3, 17 MB 1.07 and 0.69, 4.2 MB 0.35 and 0.26; to a used one 85 MB
// 5.0 and 3.5; from the host 85 MB 6.5 and 3.1.  The slots are made in about 4 ms.
#include "hostcopy.cuh"

#include <algorithm>
#include <cstring>
#include <thread>

namespace wg {

static bool make_slots(HostCopy* h) {
    if (h->pin) return true;
    if (h->off) return false;
    bool ok = cudaMallocHost((void**)&h->pin, 2 * HC_LANES * HC_CHUNK) == cudaSuccess;
    if (!ok) h->pin = nullptr;
    for (int t = 0; ok && t < HC_LANES; ++t) {
        ok = cudaStreamCreateWithFlags(&h->st[t], cudaStreamNonBlocking) == cudaSuccess;
        for (int q = 0; ok && q < 2; ++q) ok = cudaEventCreateWithFlags(&h->ev[t][q], cudaEventDisableTiming) == cudaSuccess;
    }
    if (!ok) {
        cudaGetLastError();
        host_copy_free(h);
        h->off = true;
    }
    return ok;
}

void host_copy_free(HostCopy* h) {
    for (int t = 0; t < HC_LANES; ++t) {
        for (int q = 0; q < 2; ++q)
            if (h->ev[t][q]) { cudaEventDestroy(h->ev[t][q]); h->ev[t][q] = nullptr; }
        if (h->st[t]) { cudaStreamDestroy(h->st[t]); h->st[t] = nullptr; }
    }
    if (h->pin) { cudaFreeHost(h->pin); h->pin = nullptr; }
}

// bytes [lo, hi) by lane t
static cudaError_t lane_copy(HostCopy* h, int device, int t, char* dst, const char* src, size_t lo, size_t hi,
                             cudaMemcpyKind kind) {
    cudaError_t e = cudaSetDevice(device);
    char* slot[2] = {h->pin + (size_t)(2 * t) * HC_CHUNK, h->pin + (size_t)(2 * t + 1) * HC_CHUNK};
    const bool out = kind == cudaMemcpyDeviceToHost;
    size_t held[2] = {0, 0};             // device to host: bytes on their way to the slot
    size_t at[2] = {0, 0};
    int q = 0;
    for (size_t o = lo; e == cudaSuccess && (o < hi || held[0] || held[1]); q ^= 1) {
        // the slot's last chunk
        if (held[q]) {
            if ((e = cudaEventSynchronize(h->ev[t][q])) != cudaSuccess) break;
            if (out) memcpy(dst + at[q], slot[q], held[q]);
            held[q] = 0;
        }
        if (o >= hi) continue;
        const size_t n = std::min(HC_CHUNK, hi - o);
        if (!out) memcpy(slot[q], src + o, n);
        e = cudaMemcpyAsync(out ? slot[q] : dst + o, out ? src + o : slot[q], n, kind, h->st[t]);
        if (e == cudaSuccess) e = cudaEventRecord(h->ev[t][q], h->st[t]);
        held[q] = n;
        at[q] = o;
        o += n;
    }
    const cudaError_t e2 = cudaStreamSynchronize(h->st[t]);
    return e != cudaSuccess ? e : e2;
}

static cudaError_t lanes_copy(HostCopy* h, int device, void* dst, const void* src, size_t bytes, cudaMemcpyKind kind) {
    cudaError_t e = cudaSuccess;
    const int lanes = (int)std::min<size_t>({(size_t)HC_LANES, std::max<size_t>(std::thread::hardware_concurrency(), 1),
                                             bytes / (2 * HC_CHUNK)});
    // parts of whole chunks
    const size_t part = (bytes / lanes + HC_CHUNK) / HC_CHUNK * HC_CHUNK;
    cudaError_t res[HC_LANES];
    std::thread th[HC_LANES];
    auto lane = [&](int t) {
        res[t] = lane_copy(h, device, t, (char*)dst, (const char*)src, std::min(bytes, t * part), std::min(bytes, (t + 1) * part), kind);
    };
    for (int t = 1; t < lanes; ++t) {
        try {
            th[t] = std::thread(lane, t);
        } catch (...) {                  // no thread to be had: this one does its part
            lane(t);
        }
    }
    lane(0);
    for (int t = 0; t < lanes; ++t) {
        if (th[t].joinable()) th[t].join();
        if (e == cudaSuccess) e = res[t];
    }
    return e;
}

cudaError_t host_copy(HostCopy* h, int device, void* dst, const void* src, size_t bytes, cudaMemcpyKind kind,
                      cudaStream_t s) {
    if (bytes < HC_MIN) return cudaMemcpyAsync(dst, src, bytes, kind, s);
    cudaPointerAttributes pa;
    const void* host = kind == cudaMemcpyDeviceToHost ? dst : src;
    int current = device;
    cudaGetDevice(&current);
    if (current != device) cudaSetDevice(device);
    const bool known = cudaPointerGetAttributes(&pa, host) == cudaSuccess;
    if (!known) cudaGetLastError();
    const bool staged = known && pa.type == cudaMemoryTypeUnregistered && make_slots(h);
    cudaError_t e = staged ? cudaStreamSynchronize(s) : cudaSuccess;
    if (staged && e == cudaSuccess) e = lanes_copy(h, device, dst, src, bytes, kind);
    if (current != device) cudaSetDevice(current);
    if (staged) return e;
    return cudaMemcpyAsync(dst, src, bytes, kind, s);
}

}  // namespace wg
