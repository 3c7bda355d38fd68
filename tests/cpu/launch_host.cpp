// Host-side check of fa::launch_dependent (csrc/host_common.h) on a stand-in for the CUDA runtime whose launches
// fail: the error must come back as FA_ERR_CUDA and must not stay pending, where the caller's next
// cudaGetLastError() would take it for its own.  Prints "ok" and exits 0, or prints what failed and
// exits 1.  Built and run by tests/test_launch_cpu.py.
#include <cstdio>

#include "host_common.h"

static cudaError_t g_next = cudaSuccess, g_pending = cudaSuccess;
static int g_launches = 0, g_attrs = 0;
static const char* g_noted = "";

extern "C" cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* config, const void*, void**) {
    g_launches++;
    g_attrs = (int)config->numAttrs;
    if (g_next != cudaSuccess) g_pending = g_next;
    return g_next;
}
extern "C" cudaError_t cudaGetLastError() {
    const cudaError_t e = g_pending;
    g_pending = cudaSuccess;
    return e;
}
namespace fa {
int note_cuda_error(cudaError_t, const char* where) {
    g_noted = where;
    return FA_ERR_CUDA;
}
}  // namespace fa

static void kernel(int, float) {}

#define CHECK(cond)                                                        \
    do {                                                                   \
        if (!(cond)) { std::printf("FAILED line %d: %s\n", __LINE__, #cond); return 1; } \
    } while (0)

int main() {
    CHECK(fa::launch_dependent(kernel, 1, 32, 0, nullptr, 1, 1, 2.0f) == FA_OK);
    CHECK(g_launches == 1 && g_attrs == 1 && g_pending == cudaSuccess);
    CHECK(fa::launch_dependent(kernel, 4, 32, 0, nullptr, 4, 1, 2.0f) == FA_OK);
    CHECK(g_launches == 2 && g_attrs == 2);
    for (cudaError_t e : {cudaErrorInvalidConfiguration, cudaErrorLaunchOutOfResources}) {
        g_next = e;
        g_noted = "";
        CHECK(fa::launch_dependent(kernel, 1, 32, 0, nullptr, 1, 1, 2.0f) == FA_ERR_CUDA);
        CHECK(g_noted[0] != 0);
        CHECK(g_pending == cudaSuccess);                   // nothing left for the caller's next check
    }
    std::printf("ok\n");
    return 0;
}
