// Grid barrier of the persistent kernels: all CTAs of a cooperative launch (co-resident), one arrival
// counter in global memory and a bounded poll by one thread per CTA.
#pragma once
#include "pic_kernels.h"

namespace pic {

struct GridWait {
    unsigned* arrived;  // arrivals so far
    long long polls;    // polls of a wait before it gives up
    unsigned* err;      // the world's device error word
    int* fail;          // set when a wait ran out
};
// false when the other CTAs did not arrive in time.  Global writes of any thread of the grid before it
// are seen by L2 reads (__ldcg) of any thread after it.  target: the arrivals that end this barrier,
// zero-initialised by the caller; s_fail: a shared flag, zero until a wait ran out.
__device__ __forceinline__ bool grid_barrier(const GridWait& w, unsigned& target, int* s_fail) {
    target += gridDim.x;
    __syncthreads();
    if (threadIdx.x == 0) {
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(w.arrived) : "memory");
        bool ok = false;
        for (long long it = 0; it < w.polls && !ok; it++) {
            unsigned c;
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(c) : "l"(w.arrived) : "memory");
            ok = (int)(c - target) >= 0;
        }
        if (!ok) *s_fail = 1;
    }
    __syncthreads();
    return *s_fail == 0;
}

}  // namespace pic
