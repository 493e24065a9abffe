// The wait of a CTA on the progress that another CTA of its launch publishes in global memory, and the
// publication. Every wait is bounded: after its polls it raises an error flag, which ends the launch's other
// waits too.
#pragma once

namespace bd {

constexpr unsigned kChainPolls = 1u << 22;   // polls of ~0.7 us: about 3 s, then an error

__device__ __forceinline__ int ld_acquire(const int* p) {
    int v;
    asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_release(int* p, int v) {
    asm volatile("st.release.gpu.global.s32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// Waits until *p > plane; false when the polls run out or another wait already has.
__device__ __forceinline__ bool chain_wait(const int* p, int plane, int& seen, int* err,
                                           unsigned polls = kChainPolls) {
    for (unsigned it = 0; it < polls; ++it) {
        seen = ld_acquire(p);
        if (seen > plane) return true;
        if ((it & 255u) == 255u && ld_acquire(err) != 0) return false;
    }
    atomicExch(err, 1);
    return false;
}

}  // namespace bd
