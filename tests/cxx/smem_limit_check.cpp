// Checks csrc/smem_limit.h against a stand-in of the runtime calls it makes: whatever
// another thread does between any two of them, no launch that was allowed is refused.
// Prints "ok" or what failed.
#include <cstdio>

#include "smem_limit.h"

static const int kOptin = 232448, kStatic = 48;
static int limit_ = 0;                 // the kernel's
static int calls_ = 0, interrupt_ = -1;  // the other thread runs before this call
static size_t other_ = 0;

static void step() {
    if (calls_++ == interrupt_) {
        interrupt_ = -1;
        const int at = calls_;
        pdipc::allow_smem(nullptr, other_);
        calls_ = at;
    }
}
extern "C" {
cudaError_t cudaGetDevice(int* d) {
    step();
    *d = 0;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
    step();
    if (a != cudaDevAttrMaxSharedMemoryPerBlockOptin) return cudaErrorInvalidValue;
    *v = kOptin;
    return cudaSuccess;
}
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes* fa, const void*) {
    step();
    *fa = cudaFuncAttributes();
    fa->sharedSizeBytes = kStatic;
    fa->maxDynamicSharedSizeBytes = limit_;
    return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute a, int v) {
    step();
    if (a != cudaFuncAttributeMaxDynamicSharedMemorySize || v < 0 || v + kStatic > kOptin) return cudaErrorInvalidValue;
    limit_ = v;
    return cudaSuccess;
}
}

int main() {
    const size_t sizes[] = {0, 1000, 49152, 100000, (size_t)(kOptin - kStatic)};
    for (size_t mine : sizes)
        for (size_t other : sizes)
            for (int at = -1; at < 6; ++at) {
                limit_ = 49152;
                calls_ = 0;
                interrupt_ = at;
                other_ = other;
                if (pdipc::allow_smem(nullptr, mine) != cudaSuccess || (size_t)limit_ < mine ||
                    (at >= 0 && interrupt_ < 0 && (size_t)limit_ < other)) {
                    printf("%zu bytes, %zu on another thread before call %d: limit %d\n", mine, other, at, limit_);
                    return 1;
                }
            }
    if (pdipc::allow_smem(nullptr, kOptin - kStatic + 1) == cudaSuccess) {
        printf("more than the device has was allowed\n");
        return 1;
    }
    printf("ok\n");
    return 0;
}
