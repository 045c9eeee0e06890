// Number density of one species without any device allocation.
//
// Some callers cannot allocate device memory: plugins whose host application owns all device
// memory through its own allocator (a cudaMalloc of theirs would bypass that allocator's
// accounting and limits), and real-time loops that forbid allocation after start-up because an
// allocation can block for an unbounded time.  They still own the particle arrays and the
// output field, and pass them in.  The only working memory this entry point needs -- the 64-bit
// fixed-point accumulator of one node field -- lives in the file-scope device array below, sized
// for kNoAllocMaxNodes nodes.  Every GPU that loads the library holds it (8 MiB) until the
// process exits.
//
// The array name is only a host-side stand-in for a device address; the real address is
// looked up with cudaGetSymbolAddress once per device, with that device current, on the first
// call made on the device.  That first call should therefore happen before any stream
// capture.  All calls share the one array and it keeps the last call's contents, so each call
// clears the part it uses first, and calls that overlap on the GPU (different streams, or
// different host threads on the same device) race on it.
#include <algorithm>
#include <cstdio>
#include <mutex>
#include "../../include/pic_gb300.h"
#include "pic_kernels.h"

namespace pic {

constexpr int kNoAllocMaxNodes = 1 << 20;  // 64 x 64 x 256 nodes
constexpr int kNoAllocMaxDevices = 64;

static __device__ __align__(256) unsigned long long g_noalloc_acc[kNoAllocMaxNodes];

// Eight corner contributions per particle, 64-bit fixed point (same weights and rounding as the deposit of
// the fused push kernel).  A thread takes a run of consecutive particles and holds its cell's eight sums in
// registers until the cell changes; a step to the next cell in x keeps the four sums that the two share.
// Integer sums: no order or grouping changes a bit.
//
// One atomic and one 64-bit conversion per corner and particle bound this before (the conversions, 2 a clock
// and SM, 140 us of 270 for 10 M particles; now 32-bit ones wherever they give the same).  A warp stages the
// next kPiece particles of its 32 runs with cp.async while it sums the ones before, so that the reads are
// whole sectors although each thread walks its own run.  What bounds it now is the instructions (180 a warp
// and turn; the 320 MB would take 45 us), and for particles in no order the atomics.  The whole call: 10 M
// particles in cell order, 10 to a cell, 300 -> 97 us; 8 M of 120 to a cell 717 -> 71; 6 M in no order 256 -> 182
// (278 with each thread's sums straight to the accumulator).
constexpr int kDepThr = 128, kPiece = 4;
constexpr int kQueue = 88;       // entries a warp holds: 64 of one particle each lane, 24 waiting
constexpr int kDepRun = 32;      // longest run: 32 x 32 particles of a warp lie within 16 KB
constexpr int kDepBlocks = 152 * 6;  // six per SM
__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src));
}
__device__ __forceinline__ void cp_async4(void* dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src));
}
__global__ void __launch_bounds__(kDepThr, 6) k_noalloc_deposit(GridDev g, const float4* __restrict__ pos,
                                                                const float4* __restrict__ vel, long n, int run,
                                                                float scale, unsigned long long* acc) {
    static_assert(kPiece == 4, "the swizzles below");
    constexpr int kSet = 32 * kPiece;  // staged particles of a warp
    __shared__ float4 sp[kDepThr / 32][2][kSet];
    __shared__ float sw[kDepThr / 32][2][kSet];
    __shared__ __align__(16) unsigned long long qv[kDepThr / 32][kQueue][4];
    __shared__ int qb[kDepThr / 32][kQueue];
    const int nij = g.ni * g.nj, lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
    const long per_warp = 32l * run, step = (long)gridDim.x * (kDepThr / 32) * per_warp;
    // Sums that are complete wait in the warp's queue, four corners (a face in x) an entry, until all lanes
    // write eight entries at a time: the two faces of a cell share sectors, and threads that end their runs
    // at different particles do not take the atomics' instructions one after the other.
    int held = 0;
    const int corner = ((lane & 1) ? g.ni : 0) + ((lane & 2) ? nij : 0);
    auto drain = [&]() {
        __syncwarp();
        for (int h = lane >> 2; h < held; h += 8) atomicAdd(&acc[(unsigned)(qb[wp][h] + corner)], qv[wp][h][lane & 3]);
        held = 0;
        __syncwarp();
    };
    auto queue = [&](bool out, bool all, int base, const unsigned long long* lo, const unsigned long long* hi) {
        const unsigned mo = __ballot_sync(0xffffffffu, out);
        if (!mo) return;
        const unsigned ma = __ballot_sync(0xffffffffu, all), below = (1u << lane) - 1u;
        const int at = held + __popc(mo & below) + __popc(ma & below);
        if (out) {
            ulonglong2* t = reinterpret_cast<ulonglong2*>(qv[wp][at]);
            t[0] = make_ulonglong2(lo[0], lo[1]);
            t[1] = make_ulonglong2(lo[2], lo[3]);
            qb[wp][at] = base;
            if (all) {
                t[2] = make_ulonglong2(hi[0], hi[1]);
                t[3] = make_ulonglong2(hi[2], hi[3]);
                qb[wp][at + 1] = base + 1;
            }
        }
        held += __popc(mo) + __popc(ma);
        if (held > kQueue - 64) drain();
    };
    for (long w0 = ((long)blockIdx.x * (kDepThr / 32) + wp) * per_warp; w0 < n; w0 += step) {
        // particles off .. off + kPiece - 1 of the runs, four lanes a run; slots swizzled for the reads below
        const float4 *pw = pos + w0, *vw = vel + w0;
        const int own = lane >> 2, q4 = lane & 3, most = n - w0 < per_warp ? (int)(n - w0) : (int)per_warp;
        auto stage = [&](int off, int buf) {
            float4* dp = &sp[wp][buf][(lane & ~3) + (q4 ^ ((lane >> 3) & 3))];
#pragma unroll
            for (int u = 0; u < kPiece; u++) {
                const int x = (own + 8 * u) * run + off + q4;
                if (off + q4 < run && x < most) {
                    cp_async16(dp + 32 * u, pw + x);
                    cp_async4(&sw[wp][buf][32 * u + (lane ^ u)], &vw[x].w);
                }
            }
            asm volatile("cp.async.commit_group;");
        };
        const long left = n - (w0 + (long)lane * run);
        const int m = left < run ? (left > 0 ? (int)left : 0) : run;  // particles of this thread
        unsigned long long lo[4] = {0, 0, 0, 0}, hi[4] = {0, 0, 0, 0};  // corners x0, x1: (y, z) = 00, 10, 01, 11
        int cell = -1, base = 0;
        stage(0, 0);
        for (int off = 0, buf = 0; off < run; off += kPiece, buf ^= 1) {
            if (off + kPiece < run) {
                stage(off + kPiece, buf ^ 1);
                asm volatile("cp.async.wait_group 1;" ::: "memory");
            } else {
                asm volatile("cp.async.wait_group 0;" ::: "memory");
            }
            __syncwarp();
#pragma unroll 1
            for (int q = 0; q < kPiece; q++) {
                const float4 ps = sp[wp][buf][lane * kPiece + (q ^ ((lane >> 1) & 3))];
                const int c = __float_as_int(ps.w), i = c & 511, j = (c >> 9) & 511, k = c >> 18;
                // not a removed particle, and a cell of this grid
                const bool live = off + q < m && c >= 0 && i < g.ci && j < g.cj && k < g.ck;
                const int b = cell_base_node(g, i, j, k);
                const bool turn = live && c != cell, out = turn && cell >= 0, all = out && b != base + 1;
                queue(out, all, base, lo, hi);
                if (turn) {
#pragma unroll
                    for (int x = 0; x < 4; x++) {
                        lo[x] = out && !all ? hi[x] : 0ull;
                        hi[x] = 0ull;
                    }
                    cell = c;
                    base = b;
                }
                if (!live) continue;
                const float w = sw[wp][buf][lane * kPiece + (q ^ ((lane >> 3) & 3))];
                const float wx1 = ps.x, wx0 = 1.f - ps.x, wy1 = ps.y, wy0 = 1.f - ps.y, wz1 = ps.z, wz0 = 1.f - ps.z;
                const float s = w * scale;
                const float s00 = s * wx0 * wy0, s10 = s * wx1 * wy0, s01 = s * wx0 * wy1, s11 = s * wx1 * wy1;
                const float v[8] = {s00 * wz0, s01 * wz0, s00 * wz1, s01 * wz1, s10 * wz0, s11 * wz0, s10 * wz1, s11 * wz1};
                unsigned most = 0;
#pragma unroll
                for (int x = 0; x < 8; x++) most = max(most, __float_as_uint(v[x]));
                if (most < __float_as_uint(0x1p32f)) {  // all in [0, 2^32): 32-bit conversions, the usual case
#pragma unroll
                    for (int x = 0; x < 4; x++) {
                        lo[x] += __float2uint_rn(v[x]);
                        hi[x] += __float2uint_rn(v[x + 4]);
                    }
                } else {
#pragma unroll 1
                    for (int x = 0; x < 4; x++) {
                        const float a = x == 0 ? v[0] : x == 1 ? v[1] : x == 2 ? v[2] : v[3];
                        const float b = x == 0 ? v[4] : x == 1 ? v[5] : x == 2 ? v[6] : v[7];
                        const unsigned long long ta = __float2ull_rn(a), tb = __float2ull_rn(b);
#pragma unroll
                        for (int y = 0; y < 4; y++) {
                            lo[y] += y == x ? ta : 0ull;
                            hi[y] += y == x ? tb : 0ull;
                        }
                    }
                }
            }
            __syncwarp();  // the buffer is staged again in the next turn
        }
        queue(cell >= 0, cell >= 0, base, lo, hi);
    }
    drain();
}

// den = accumulated weight / node volume, periodic copies folded onto index 0.  f: 1 / (scale x volume) of a
// node on 0, 1, 2, 3 walls in FP64 (powers of two apart): FP64 runs at 2 operations a clock and SM here, so
// that a division per thread took most of the pass.
struct DenFactors {
    double f[4];
    __device__ __forceinline__ double at(int w) const { return w < 2 ? (w ? f[1] : f[0]) : (w == 2 ? f[2] : f[3]); }
};
__global__ void k_noalloc_finalize(GridDev g, const unsigned long long* __restrict__ acc, DenFactors df,
                                   float* __restrict__ den) {
    const int nn[3] = {g.ni, g.nj, g.nk}, stride[3] = {1, g.ni, g.ni * g.nj};
    for (int n = blockIdx.x * blockDim.x + threadIdx.x; n < g.nv; n += gridDim.x * blockDim.x) {
        int ijk[3];
        int r = n / g.ni;
        ijk[0] = n - r * g.ni;
        ijk[2] = r / g.nj;
        ijk[1] = r - ijk[2] * g.nj;
        bool alias = false;
        unsigned fold = 0;
        int walls = 0;
        for (int d = 0; d < 3; d++) {
            if (g.periodic[d]) {
                if (ijk[d] == nn[d] - 1) alias = true;
                if (ijk[d] == 0) fold |= 1u << d;
            } else if (ijk[d] == 0 || ijk[d] == nn[d] - 1) {
                walls++;
            }
        }
        if (alias) continue;
        unsigned long long tot = 0;
        for (unsigned m = 0; m < 8; m++) {
            if (m & ~fold) continue;
            int node = n;
            for (int d = 0; d < 3; d++)
                if (m & (1u << d)) node += (nn[d] - 1) * stride[d];
            tot += acc[node];
        }
        float v = (float)((double)tot * df.at(walls));
        for (unsigned m = 0; m < 8; m++) {
            if (m & ~fold) continue;
            int node = n;
            for (int d = 0; d < 3; d++)
                if (m & (1u << d)) node += (nn[d] - 1) * stride[d];
            den[node] = v;
        }
    }
}

namespace {
std::mutex g_noalloc_mutex;
void* g_noalloc_ptr[kNoAllocMaxDevices] = {};
}  // namespace

}  // namespace pic

using namespace pic;

extern "C" int pic_number_density_noalloc(int ni, int nj, int nk, const double* x0, const double* xm,
                                          const int* periodic, const void* pos4, const void* vel4, long n,
                                          double scale, float* den_out, void* stream) {
    long long nv = (long long)ni * nj * nk;
    if (!x0 || !xm || (n > 0 && (!pos4 || !vel4)) || !den_out || n < 0 || !(scale > 0))
        return set_last_error(PIC_ERR_ARG, "pic_number_density_noalloc: null array, negative count or scale <= 0");
    // the packed particle cell keeps 9 bits for i and j and 13 for k (pic_world_create's limits)
    if (ni < 2 || nj < 2 || nk < 2 || ni - 1 > kCellMaxIJ || nj - 1 > kCellMaxIJ || nk - 1 > kCellMaxK)
        return set_last_error(PIC_ERR_ARG, "pic_number_density_noalloc: grid must have 2..513 x 2..513 x 2..8193 nodes");
    if (nv > kNoAllocMaxNodes) {
        char msg[160];
        snprintf(msg, sizeof(msg), "pic_number_density_noalloc: %lld nodes exceed the %d-node accumulator", nv,
                 kNoAllocMaxNodes);
        return set_last_error(PIC_ERR_ARG, msg);
    }
    for (int d = 0; d < 3; d++)
        if (!(xm[d] > x0[d])) return set_last_error(PIC_ERR_ARG, "pic_number_density_noalloc: xm must exceed x0");
    {
        const int nn3[3] = {ni, nj, nk};
        for (int d = 0; d < 3; d++)  // as pic_world_set_boundaries
            if (periodic && periodic[d] && nn3[d] < 4)
                return set_last_error(PIC_ERR_ARG, "pic_number_density_noalloc: periodic axis needs at least 4 nodes");
    }
    // the deposit scales in FP32; the finalize divides by the same FP32 value
    const float fscale = (float)scale;
    if (!(fscale > 0.f) || !(fscale < 3.0e38f))
        return set_last_error(PIC_ERR_ARG, "pic_number_density_noalloc: scale is not a finite FP32 value");
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kNoAllocMaxDevices)
        return set_last_error(PIC_ERR_CUDA, "pic_number_density_noalloc: no current CUDA device");
    void* acc = nullptr;
    {
        // first call on this device: look up the device address of the file-scope array
        std::lock_guard<std::mutex> lock(g_noalloc_mutex);
        if (!g_noalloc_ptr[dev]) {
            void* p = nullptr;
            if (cudaGetSymbolAddress(&p, g_noalloc_acc) != cudaSuccess || !p)
                return set_last_error(PIC_ERR_CUDA, "pic_number_density_noalloc: cudaGetSymbolAddress failed");
            g_noalloc_ptr[dev] = p;
        }
        acc = g_noalloc_ptr[dev];
    }
    GridDev g{};
    g.ni = ni;
    g.nj = nj;
    g.nk = nk;
    g.ci = ni - 1;
    g.cj = nj - 1;
    g.ck = nk - 1;
    g.nv = (int)nv;
    g.nc = g.ci * g.cj * g.ck;
    int nn[3] = {ni, nj, nk};
    for (int d = 0; d < 3; d++) {
        g.x0[d] = x0[d];
        g.xm[d] = xm[d];
        g.dxd[d] = (xm[d] - x0[d]) / (nn[d] - 1);
        g.dx[d] = (float)g.dxd[d];
        g.inv_dx[d] = (float)(1.0 / g.dxd[d]);
        g.periodic[d] = periodic ? (periodic[d] != 0) : 0;
    }
    cudaStream_t s = (cudaStream_t)stream;
    if (cudaMemsetAsync(acc, 0, sizeof(unsigned long long) * nv, s) != cudaSuccess)
        return set_last_error(PIC_ERR_CUDA, "pic_number_density_noalloc: clearing the accumulator failed");
    // launched through cudaLaunchKernel, whose return value is this launch's own status: an error
    // the caller left pending before this call is neither reported nor cleared here
    unsigned long long* accp = (unsigned long long*)acc;
    if (n > 0) {
        // equal runs for all threads of a full grid in as few turns as kDepRun allows, of whole pieces
        const long blocks = std::min<long>((n + kDepThr - 1) / kDepThr, kDepBlocks), thr = blocks * kDepThr;
        const long turns = (n + thr * kDepRun - 1) / (thr * kDepRun);
        int run = (int)((n + thr * turns - 1) / (thr * turns));
        if (run > kPiece) run = (run + kPiece - 1) / kPiece * kPiece;
        const float4* p4 = (const float4*)pos4;
        const float4* v4 = (const float4*)vel4;
        void* args[] = {&g, &p4, &v4, &n, &run, (void*)&fscale, &accp};
        if (cudaLaunchKernel((const void*)k_noalloc_deposit, dim3((unsigned)blocks), dim3(kDepThr), args, 0, s) !=
            cudaSuccess)
            return set_last_error(PIC_ERR_CUDA, "pic_number_density_noalloc: deposit launch failed");
    }
    int fb = (int)((nv + 255) / 256);
    if (fb > 4096) fb = 4096;
    const unsigned long long* caccp = accp;
    DenFactors df;
    df.f[0] = (1.0 / (double)fscale) * (1.0 / (g.dxd[0] * g.dxd[1] * g.dxd[2]));
    for (int d = 0; d < 3; d++) df.f[d + 1] = 2.0 * df.f[d];
    void* fargs[] = {&g, &caccp, &df, &den_out};
    if (cudaLaunchKernel((const void*)k_noalloc_finalize, dim3((unsigned)fb), dim3(256), fargs, 0, s) != cudaSuccess)
        return set_last_error(PIC_ERR_CUDA, "pic_number_density_noalloc: finalize launch failed");
    return PIC_OK;
}
