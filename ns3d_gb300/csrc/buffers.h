// buffers.h -- errors, and the ownership of device and host staging memory.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <stdexcept>
#include <string>
#include <vector>

#include "../../include/ns3d_capi.h"

namespace ns3d {

struct CudaError : std::runtime_error {
    cudaError_t code;
    CudaError(cudaError_t e, const char *expr, const char *file, int line)
        : std::runtime_error(std::string(cudaGetErrorString(e)) + " in " + expr + " (" + file + ":" +
                             std::to_string(line) + ")"),
          code(e) {}
};

struct ApiError : std::runtime_error {
    int code;
    ApiError(int c, const std::string &m) : std::runtime_error(m), code(c) {}
};

}  // namespace ns3d

#define NS3D_CUDA_CHECK(expr)                                                          \
    do {                                                                               \
        cudaError_t _e = (expr);                                                       \
        if (_e != cudaSuccess) throw ns3d::CudaError(_e, #expr, __FILE__, __LINE__);   \
    } while (0)

namespace ns3d {

// Device memory of the library: one stream-ordered pool per device, kept
// reserved between solves (no cudaMalloc / cudaFree, which synchronize the
// whole device and would stall every other solve running in the process).
cudaMemPool_t device_pool();

// Device array allocated on a stream from the library pool and freed on the
// same stream (stream-ordered: it may be released while work that uses it
// is still queued on that stream).
template <class T>
struct DBuf {
    T *p = nullptr;
    size_t n = 0;
    cudaStream_t st_ = nullptr;
    DBuf() = default;
    DBuf(const DBuf &) = delete;
    DBuf &operator=(const DBuf &) = delete;
    ~DBuf() { release(); }
    void alloc(size_t count, cudaStream_t st) {
        release();
        n = count;
        st_ = st;
        if (count == 0) return;
        cudaError_t e = cudaMallocFromPoolAsync((void **)&p, count * sizeof(T), device_pool(), st);
        if (e != cudaSuccess) {
            p = nullptr;
            n = 0;
            cudaGetLastError();
            throw ApiError(NS3D_ERR_OOM, "device allocation of " + std::to_string(count * sizeof(T)) + " bytes failed");
        }
    }
    void alloc_zero(size_t count, cudaStream_t st) {
        alloc(count, st);
        if (count) NS3D_CUDA_CHECK(cudaMemsetAsync(p, 0, count * sizeof(T), st));
    }
    void release() {
        if (p) cudaFreeAsync(p, st_);
        p = nullptr;
        n = 0;
    }
};

// Host staging array of the small per-solve state copies.  Pageable memory:
// a device-to-host copy into it returns once the copy is done, and freeing
// it does not synchronize the device (cudaFreeHost would).
template <class T>
struct HBuf {
    std::vector<T> v;
    T *p = nullptr;
    size_t n = 0;
    void alloc(size_t count) {
        v.assign(count, T());
        p = count ? v.data() : nullptr;
        n = count;
    }
};

// What a solve set keeps for each of its systems, in lines of type T on the
// device and in a host copy.  `cap` is the number of systems there is room
// for in both; after an allocation that failed there is room for none, so
// the next set-up tries again.
template <class T>
struct StateBuf {
    DBuf<T> dev;
    HBuf<T> host;
    int cap = 0;
    // room for `count` systems, which take `bytes`
    void reserve(int count, size_t bytes, cudaStream_t st) {
        if (count <= cap) return;
        cap = 0;
        const size_t lines = (bytes + sizeof(T) - 1) / sizeof(T);
        dev.alloc_zero(lines, st);
        host.alloc(lines);
        cap = count;
    }
};

}  // namespace ns3d
