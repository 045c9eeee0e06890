// Grid barrier of the persistent kernels: all CTAs of a cooperative launch (co-resident), one arrival
// counter in global memory and a bounded poll by one thread per CTA.
#pragma once
#include "pic_ff.cuh"
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

constexpr int kMostCtas = 512;  // CTAs whose partial sums a launch holds
// what the CTAs of a launch share, the counter zero at launch
struct GridSync {
    unsigned arrived;
    unsigned pad[31];
    float2 part[4][kMostCtas];  // float-float partials: d.q, then the three sums after the update
};
// a + t, the high parts by TwoSum, the low parts collected (normalised once at the end of a sum)
__device__ __forceinline__ FF ff_gather(FF a, FF t) {
    const FF s = two_sum(a.hi, t.hi);
    return FF{s.hi, a.lo + (t.lo + s.lo)};
}
constexpr int kAtOnce = 5;  // partials a lane reads at once: 152 CTAs in one go
// Sums of N per-thread values over the grid, in every lane of warp 0 of every CTA: FP32 within a warp,
// float-float over the warps and the CTAs, in a fixed order; passes one grid barrier (false: it failed).
// part: the N slots of this sum, not read by anyone since the last barrier but one.
template <int N, int NT>
__device__ __forceinline__ bool grid_total(const float (&v)[N], float (*wsum)[NT / 32], float2 (*part)[kMostCtas],
                                           const GridWait& w, unsigned& target, int* s_fail, FF (&out)[N]) {
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
    float x[N];
#pragma unroll
    for (int c = 0; c < N; c++) x[c] = v[c];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int c = 0; c < N; c++) x[c] += __shfl_xor_sync(0xffffffffu, x[c], o);
    if (lane == 0)
#pragma unroll
        for (int c = 0; c < N; c++) wsum[c][wp] = x[c];
    auto tree = [&]() {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
#pragma unroll
            for (int c = 0; c < N; c++)
                out[c] = ff_gather(out[c], FF{__shfl_xor_sync(0xffffffffu, out[c].hi, o),
                                              __shfl_xor_sync(0xffffffffu, out[c].lo, o)});
#pragma unroll
        for (int c = 0; c < N; c++) out[c] = two_sum(out[c].hi, out[c].lo);
    };
    __syncthreads();
    if (wp == 0) {
#pragma unroll
        for (int c = 0; c < N; c++) out[c] = FF{lane < NT / 32 ? wsum[c][lane] : 0.f, 0.f};
        tree();
        if (lane == 0)
#pragma unroll
            for (int c = 0; c < N; c++) __stcg(&part[c][blockIdx.x], make_float2(out[c].hi, out[c].lo));
    }
    const bool ok = grid_barrier(w, target, s_fail);
    if (wp == 0) {
#pragma unroll
        for (int c = 0; c < N; c++) out[c] = FF{0.f, 0.f};
        for (int b0 = lane; b0 < (int)gridDim.x; b0 += 32 * kAtOnce) {
            float2 t[kAtOnce][N];  // every load in flight before the first is used: one L2 latency
#pragma unroll
            for (int u = 0; u < kAtOnce; u++)
#pragma unroll
                for (int c = 0; c < N; c++)
                    t[u][c] = b0 + 32 * u < (int)gridDim.x ? __ldcg(&part[c][b0 + 32 * u]) : make_float2(0.f, 0.f);
#pragma unroll
            for (int u = 0; u < kAtOnce; u++)
#pragma unroll
                for (int c = 0; c < N; c++) out[c] = ff_gather(out[c], FF{t[u][c].x, t[u][c].y});
        }
        tree();
    }
    return ok;
}
__device__ __forceinline__ float ff_ratio(FF a, FF b) {  // a / b rounded to FP32
    const float q = a.hi / b.hi;
    const float rem = fmaf(-q, b.hi, a.hi) + (a.lo - q * b.lo);
    return q + rem / b.hi;
}


}  // namespace pic
