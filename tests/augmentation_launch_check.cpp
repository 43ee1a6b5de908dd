// The host side of the augmentation's launches, with the runtime's calls that would
// reach a device replaced: nothing here touches a GPU, present or not.
#include "augmentation.h"

#include <cstdio>

static int launches = 0;
static cudaError_t limit_status = cudaSuccess, launch_status = cudaSuccess;

extern "C" {
cudaError_t cudaGetDevice(int *device) {
    *device = 0;
    return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void *, cudaFuncAttribute, int) {
    return limit_status;
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *, const void *, void **) {
    ++launches;
    return launch_status;
}
cudaError_t cudaLaunchKernel(const void *, dim3, dim3, void **, size_t, cudaStream_t) {
    ++launches;
    return launch_status;
}
cudaError_t cudaDeviceGetAttribute(int *value, cudaDeviceAttr, int) {
    *value = 148;
    return cudaSuccess;
}
cudaError_t cudaPeekAtLastError() {
    return launch_status;
}
}

namespace vitb200 {
unsigned long long g_kernel_launches = 0;
}

#define CHECK(condition)                                              \
    if (!(condition)) {                                               \
        printf("line %d: %s\n", __LINE__, #condition);                \
        return 1;                                                     \
    }

int main() {
    using namespace vitb200;
    // Scratch for every batch that does not go plane by plane, one with more planes
    // than a grid has blocks among them.
    CHECK(augmentation_scratch_bytes(2048, 3, 28, 28) == 0);
    CHECK(augmentation_scratch_bytes(2, 1, 160, 160) == 0);
    CHECK(augmentation_scratch_bytes(2, 1, 161, 160) > 0);
    CHECK(augmentation_scratch_bytes(0x7fffffffu, 1, 1, 1) == 0);
    CHECK(augmentation_scratch_bytes(0x80000000u, 1, 1, 1) > 0);
    CHECK(augmentation_scratch_bytes(0x40000000u, 2, 1, 1) > 0);
    // A kernel that cannot be launched is reported, every time.
    AugmentationSettings settings = {};
    settings.max_shift_pixels = 2.0f;
    settings.noise_standard_deviation = 0.01f;
    float *somewhere = nullptr;
    auto apply = [&](size_t size) {
        launches = 0;
        return launch_augmentation(settings, nullptr, somewhere, somewhere, somewhere, 2,
                                   1, size, size, nullptr);
    };
    limit_status = cudaErrorInvalidValue;   // planes above 40 KiB ask for more
    CHECK(!apply(100) && launches == 0);
    CHECK(!apply(100) && launches == 0);
    CHECK(apply(28) && launches == 1);
    limit_status = cudaSuccess;
    CHECK(apply(100) && launches == 1);
    CHECK(apply(200) && launches > 1);
    launch_status = cudaErrorInvalidConfiguration;
    CHECK(!apply(28) && !apply(100) && !apply(200));
    return 0;
}
