// What common.cuh and geometry.cuh need of CUDA to compile as host C++: declaration
// keywords and the few intrinsics their inline functions name (none is called here).
#pragma once
#include <cuda_runtime.h>

template <typename T>
inline T __ldg(const T* p) {
    return *p;
}
template <typename T>
inline T __shfl_xor_sync(unsigned, T v, int) {
    return v;
}
template <typename T>
inline T atomicMin(T* p, T v) {
    const T old = *p;
    if (v < old) *p = v;
    return old;
}
inline unsigned __float_as_uint(float v) {
    unsigned u;
    __builtin_memcpy(&u, &v, sizeof u);
    return u;
}
inline long long __double_as_longlong(double v) {
    long long u;
    __builtin_memcpy(&u, &v, sizeof u);
    return u;
}
inline float __double2float_rn(double v) { return (float)v; }
