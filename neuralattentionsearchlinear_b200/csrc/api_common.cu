// Error plumbing shared by every C-ABI entry point: a thread-local message buffer
// read through natsl_last_error(), and a launch check that maps CUDA errors to a
// negative status instead of aborting.
#include <stdarg.h>
#include <stdio.h>

#include "common.cuh"
#include "../../include/natsl_b200.h"

namespace natsl {

static thread_local char g_err[512] = "";

void set_error(const char* fmt, ...) {
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(g_err, sizeof(g_err), fmt, ap);
    va_end(ap);
}

// Launches (each is followed by one check) of this thread since the start of its last counted call.
static thread_local int g_launches = 0;
void count_launches_from_here() { g_launches = 0; }

int check_launch(const char* what) {
    ++g_launches;
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        set_error("%s: CUDA error %d (%s)", what, (int)e, cudaGetErrorString(e));
        return NATSL_ERR_CUDA;
    }
    return NATSL_OK;
}

int check_device(const void* p, const char* what) {
    int dev = -1;
    cudaPointerAttributes at = {};
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaPointerGetAttributes(&at, p);
    if (e != cudaSuccess) {
        cudaGetLastError();
        set_error("%s: CUDA error %d (%s)", what, (int)e, cudaGetErrorString(e));
        return NATSL_ERR_CUDA;
    }
    NATSL_REQUIRE(at.type == cudaMemoryTypeDevice || at.type == cudaMemoryTypeManaged, NATSL_ERR_UNSUPPORTED,
                  "%s: a tensor is not in device memory", what);
    NATSL_REQUIRE(at.type == cudaMemoryTypeManaged || at.device == dev, NATSL_ERR_UNSUPPORTED,
                  "%s: the tensors are on device %d, the current device is %d", what, at.device, dev);
    return NATSL_OK;
}

}  // namespace natsl

extern "C" const char* natsl_last_error(void) { return natsl::g_err; }

extern "C" int natsl_call_kernels(void) { return natsl::g_launches; }

extern "C" int natsl_abi_version(void) { return NATSL_B200_ABI_VERSION; }
