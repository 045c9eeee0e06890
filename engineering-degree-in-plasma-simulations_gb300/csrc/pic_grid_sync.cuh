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
constexpr int kAtOnce = 5;  // partials a lane reads at once: 152 CTAs in one go
// sums over a warp in every lane
template <int N>
__device__ __forceinline__ void warp_total(FF (&x)[N]) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int c = 0; c < N; c++)
            x[c] = ff_gather(x[c], FF{__shfl_xor_sync(0xffffffffu, x[c].hi, o), __shfl_xor_sync(0xffffffffu, x[c].lo, o)});
#pragma unroll
    for (int c = 0; c < N; c++) x[c] = two_sum(x[c].hi, x[c].lo);
}
// One warp's sum of each of N values: value c ends in lane warp_home<N>(c).  The shuffles bound the sums of all warps
// of a CTA, so a lane hands over the half of the values that it does not keep first: 12 shuffles of 32 bits for
// three values instead of 30.
template <int N>
__device__ __forceinline__ constexpr int warp_home(int c) {
    return N == 2 ? 16 * c : 8 * c;
}
template <int N>
__device__ __forceinline__ FF warp_halved(const FF (&x)[N]) {
    static_assert(N >= 1 && N <= 3, "the steps below");
    const int lane = threadIdx.x & 31;
    auto from = [](FF v, int o) {
        return FF{__shfl_xor_sync(0xffffffffu, v.hi, o), __shfl_xor_sync(0xffffffffu, v.lo, o)};
    };
    const bool up = lane & 16, up8 = lane & 8;
    FF a = x[0];
    if (N == 1) {
        a = ff_gather(a, from(a, 16));
        a = ff_gather(a, from(a, 8));
    } else if (N == 2) {
        a = ff_gather(up ? x[N - 1] : x[0], from(up ? x[0] : x[N - 1], 16));
        a = ff_gather(a, from(a, 8));
    } else {  // value 2 goes up, then value 1
        a = ff_gather(up ? x[N - 1] : x[0], from(up ? x[0] : x[N - 1], 16));
        const FF b = ff_gather(x[N / 2], from(x[N / 2], 16));
        a = ff_gather(up8 ? b : a, from(up8 ? a : b, 8));
    }
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) a = ff_gather(a, from(a, o));
    return two_sum(a.hi, a.lo);
}
// Sums of N per-thread values over the grid, times scale, in every lane of warp 0 of every CTA, in a fixed order;
// passes one grid barrier (false: it failed).  part: the N slots of this sum, not read by anyone since the last
// barrier but one.  Float-float from the threads' values on (48 bits), since FP64 runs at two operations a clock
// and SM; only the sums of kFp32Nodes nodes at most that a thread adds first round at FP32.  Against FP64 a sum of
// |r|^2 is off by 2.6e-9 at 40 000 nodes and 7.3e-10 at 2.1 million (5.5e-9 and 8.5e-10 with FP32 over a thread and
// a warp and FP64 above, as in the launch-per-pass kernels).  scale is a power of two that brings the sum near 1: a
// warp's sum lies in FP32's range, the grid's need not.
template <int N, int NT>
__device__ __forceinline__ bool grid_total(const FF (&v)[N], const float (&scale)[N], float2 (*wsum)[NT / 32],
                                           float2 (*part)[kMostCtas], const GridWait& w, unsigned& target, int* s_fail,
                                           FF (&out)[N]) {
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
    const FF x = warp_halved(v);
#pragma unroll
    for (int c = 0; c < N; c++)
        if (lane == warp_home<N>(c)) wsum[c][wp] = make_float2(x.hi * scale[c], x.lo * scale[c]);
    __syncthreads();
    if (wp == 0) {
#pragma unroll
        for (int c = 0; c < N; c++) {
            const float2 t = lane < NT / 32 ? wsum[c][lane] : make_float2(0.f, 0.f);
            out[c] = FF{t.x, t.y};
        }
        warp_total(out);
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
        warp_total(out);
    }
    return ok;
}
}  // namespace pic
