// The shared-memory limit of a launch site on several devices, against a runtime
// of two functions: the current device, and which limits were raised where.
#include "shared_limit.h"

#include <cstdio>
#include <set>
#include <utility>

static int current_device = 0;
static bool refuse = false;
static std::set<std::pair<int, const void *>> raised;
static int calls = 0;

extern "C" cudaError_t cudaGetDevice(int *device) {
    *device = current_device;
    return cudaSuccess;
}

extern "C" cudaError_t cudaFuncSetAttribute(const void *kernel, cudaFuncAttribute, int) {
    ++calls;
    if (refuse) {
        return cudaErrorInvalidValue;
    }
    raised.insert({current_device, kernel});
    return cudaSuccess;
}

#define CHECK(condition)                                              \
    if (!(condition)) {                                               \
        printf("line %d: %s\n", __LINE__, #condition);                \
        return 1;                                                     \
    }

int main() {
    const int a = 0, b = 0;
    const void *kernels[] = {&a, &b};
    vitb200::SharedMemoryLimit limit;
    refuse = true;
    CHECK(!limit.raise(kernels, 2, 1 << 16));   // a failure is not remembered
    refuse = false;
    CHECK(limit.raise(kernels, 2, 1 << 16));
    calls = 0;
    CHECK(limit.raise(kernels, 2, 1 << 16) && calls == 0);
    for (int device : {1, 63, 64, 65, 0}) {
        current_device = device;
        CHECK(limit.raise(kernels, 2, 1 << 16));
        CHECK(raised.count({device, &a}) && raised.count({device, &b}));
    }
    return 0;
}
