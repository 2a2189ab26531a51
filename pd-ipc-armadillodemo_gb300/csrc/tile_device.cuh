// tile_device.cuh — device helpers of the tiled PD solves (pd_tile.cu, pd_tile3.cu):
// the exchange words, and the arithmetic whose rounding they share.
#pragma once

#include "kernels.cuh"
#include "tile.h"

namespace pdipc {

namespace {

__device__ __forceinline__ unsigned ld_acquire(const unsigned* p) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_release(unsigned* p, unsigned v) {
    asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ TileWord ld_word(const TileWord* p) {
    TileWord w;
    asm volatile(
        "{\n\t.reg .b128 v;\n\t"
        "ld.relaxed.gpu.global.b128 v, [%2];\n\t"
        "mov.b128 {%0, %1}, v;\n\t}"
        : "=l"(w.lo), "=l"(w.hi)
        : "l"(p)
        : "memory");
    return w;
}
__device__ __forceinline__ void st_word(TileWord* p, unsigned long long lo, unsigned long long hi) {
    asm volatile(
        "{\n\t.reg .b128 v;\n\t"
        "mov.b128 v, {%1, %2};\n\t"
        "st.relaxed.gpu.global.b128 [%0], v;\n\t}" ::"l"(p),
        "l"(lo), "l"(hi)
        : "memory");
}
// ---- thread-block cluster: the same place in another CTA's shared memory, and the
// barrier of all its threads (release, acquire: it orders the remote writes; without a
// limit, since the hardware runs the CTAs together and none leaves early) ----
__device__ __forceinline__ unsigned remote_addr(const void* p, unsigned rank) {
    unsigned r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;"
                 : "=r"(r)
                 : "r"((unsigned)__cvta_generic_to_shared(p)), "r"(rank));
    return r;
}
__device__ __forceinline__ void st_remote(unsigned addr, float x, float y) {
    asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(addr), "f"(x), "f"(y) : "memory");
}
__device__ __forceinline__ void st_remote(unsigned addr, float x) {
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(addr), "f"(x) : "memory");
}
__device__ __forceinline__ void st_remote(unsigned, double, double) {}
__device__ __forceinline__ void st_remote(unsigned, double) {}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
// ---- barrier of some of a CTA's threads, and whether any of them says so ----
__device__ __forceinline__ void half_sync(int id, int threads) {
    asm volatile("barrier.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
__device__ __forceinline__ bool half_sync_or(int id, int threads, bool v) {
    int any;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\tsetp.ne.s32 q, %1, 0;\n\tbarrier.red.or.pred p, %2, %3, q;\n\t"
        "selp.s32 %0, 1, 0, p;\n\t}"
        : "=r"(any)
        : "r"((int)v), "r"(id), "r"(threads)
        : "memory");
    return any != 0;
}
// ---- tensor memory as a store of constants: 512 columns x 128 lanes of 32 bits per
// SM, of which a warp reads and writes the 32 lanes of its quarter (warp % 4).  All
// of a warp's threads take part in each of these. ----
__device__ __forceinline__ void tmem_alloc(unsigned* where, unsigned columns) {  // one warp
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n\t"
                 "tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::"r"(
                     (unsigned)__cvta_generic_to_shared(where)),
                 "r"(columns)
                 : "memory");
}
__device__ __forceinline__ void tmem_free(unsigned base, unsigned columns) {  // one warp
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(base), "r"(columns) : "memory");
}
__device__ __forceinline__ void tmem_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tmem_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tmem_store4(unsigned addr, float4 v) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(__float_as_uint(v.x)),
                 "r"(__float_as_uint(v.y)), "r"(__float_as_uint(v.z)), "r"(__float_as_uint(v.w))
                 : "memory");
}
__device__ __forceinline__ void tmem_store_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// a load is under way until the wait that names its registers
__device__ __forceinline__ void tmem_load8(unsigned addr, unsigned (&u)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(u[0]), "=r"(u[1]), "=r"(u[2]), "=r"(u[3]), "=r"(u[4]), "=r"(u[5]), "=r"(u[6]), "=r"(u[7])
                 : "r"(addr));
}
__device__ __forceinline__ void tmem_wait8(unsigned (&u)[8]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(u[0]), "+r"(u[1]), "+r"(u[2]), "+r"(u[3]), "+r"(u[4]), "+r"(u[5]), "+r"(u[6]), "+r"(u[7]));
}
__device__ __forceinline__ void tmem_load2(unsigned addr, unsigned (&u)[2]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x2.b32 {%0, %1}, [%2];" : "=r"(u[0]), "=r"(u[1]) : "r"(addr));
}
__device__ __forceinline__ void tmem_wait2(unsigned (&u)[2]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;" : "+r"(u[0]), "+r"(u[1]));
}
__device__ __forceinline__ unsigned long long pack2(unsigned a, unsigned b) {
    return (unsigned long long)a | ((unsigned long long)b << 32);
}


// ---- the arithmetic, with its rounding spelled out: the results keep the bits
// of the launches this solve stands in for (one per sweep in the direct form, the
// band in the correction form), whatever the compiler would contract ----
__device__ __forceinline__ float fma_(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double fma_(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ float mul_(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mul_(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float add_(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double add_(double a, double b) { return __dadd_rn(a, b); }
// (1 - w) c + w ((s + b) / D): one weighted-Jacobi update; which of the two products
// is rounded by itself: the second, or the first (kept_first)
template <typename T>
__device__ __forceinline__ T jacobi(T om1, T c, T w, T s, T b, T id, bool kept_first) {
    const T t = mul_(add_(s, b), id);
    return fma_(kept_first ? w : om1, kept_first ? t : c, mul_(kept_first ? om1 : w, kept_first ? c : t));
}
template <typename T>
__device__ __forceinline__ T norm2(T x, T y, T z) {
    return fma_(z, z, fma_(x, x, mul_(y, y)));
}
// Sum2 (common.cuh) with the products it adds fused
struct Acc {
    float s = 0.f, c = 0.f;
    __device__ __forceinline__ void step(float t, float bp, float e) {
        c = add_(c, add_(add_(s, -add_(t, -bp)), e));
        s = t;
    }
    __device__ __forceinline__ void add(float x) {
        const float t = add_(s, x), bp = add_(t, -s);
        step(t, bp, add_(x, -bp));
    }
    __device__ __forceinline__ void add(float a, float b) {
        const float t = fma_(a, b, s), bp = add_(t, -s);
        step(t, bp, fma_(a, b, -bp));
    }
    __device__ __forceinline__ float value() const { return add_(s, c); }
};

template <typename T>
struct alignas(2 * sizeof(T)) Pair {
    T x, y;
};

// the values of consecutive entries of one row: 16 bytes
template <typename T>
struct alignas(16) Group {
    T v[16 / sizeof(T)];
};

template <typename S>
__device__ __forceinline__ V4<S> ldg_state(const V4<S>* p, int i) {  // written by this thread or an earlier kernel
    return p[i];
}

}  // namespace

}  // namespace pdipc
