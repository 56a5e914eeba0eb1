// Checks of a solve set's state buffers (StateBuf) when a device allocation
// fails: built with the library's buffers.h over fakes of the CUDA calls it
// makes, and run by tests/test_buffers.py.  No GPU.
#include <cstdio>
#include <cstdlib>
#include <cstring>

#include "../../ns3d_gb300/csrc/buffers.h"

static int live = 0;
static bool refuse = false;

extern "C" {
cudaError_t cudaMallocFromPoolAsync(void **p, size_t bytes, cudaMemPool_t, cudaStream_t) {
    if (refuse) return cudaErrorMemoryAllocation;
    *p = std::malloc(bytes);
    ++live;
    return cudaSuccess;
}
cudaError_t cudaFreeAsync(void *p, cudaStream_t) {
    std::free(p);
    --live;
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void *p, int v, size_t bytes, cudaStream_t) {
    std::memset(p, v, bytes);
    return cudaSuccess;
}
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t) { return "error"; }
}
namespace ns3d {
cudaMemPool_t device_pool() { return nullptr; }
}

static int failures = 0;
#define CHECK(cond)                                                  \
    do {                                                             \
        if (!(cond)) {                                               \
            std::printf("FAILED line %d: %s\n", __LINE__, #cond);   \
            ++failures;                                              \
        }                                                            \
    } while (0)

struct Line {
    unsigned char b[256];
};

int main() {
    {
        ns3d::StateBuf<Line> s;
        s.reserve(3, 1000, nullptr);
        CHECK(s.cap == 3 && s.dev.n == 4 && s.host.n == 4 && s.dev.p && s.host.p);
        const Line *p = s.dev.p;
        s.reserve(2, 700, nullptr);  // there is room
        CHECK(s.cap == 3 && s.dev.p == p);
        // growing fails: no room, and the next set-up, of any size, tries again
        refuse = true;
        for (int count : {9, 2}) {
            int code = 0;
            try {
                s.reserve(count, 300 * count, nullptr);
            } catch (const ns3d::ApiError &e) {
                code = e.code;
            }
            CHECK(code == NS3D_ERR_OOM && s.cap == 0 && !s.dev.p);
        }
        refuse = false;
        s.reserve(2, 600, nullptr);
        CHECK(s.cap == 2 && s.dev.p && s.dev.n == 3 && s.host.n == 3);
        for (size_t i = 0; i < 3 * sizeof(Line); ++i) CHECK(reinterpret_cast<unsigned char *>(s.dev.p)[i] == 0);
    }
    CHECK(live == 0);
    if (!failures) std::printf("OK\n");
    return failures != 0;
}
