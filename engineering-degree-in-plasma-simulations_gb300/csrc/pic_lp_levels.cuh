// Level views of the learned preconditioner on the device: index rules of the transfers and stencils, and
// the coarse levels of the hierarchy as one device function for persistent kernels.
#pragma once
#include <algorithm>
#include "pic_grid_sync.cuh"
#include "pic_learned.h"
#include "pic_stencil.cuh"

namespace pic {

__device__ __forceinline__ void lv_decode(const LView& v, unsigned idx, int& x, int& y, int& z) {
    unsigned t = fdiv(idx, v.fx);
    x = (int)(idx - t * (unsigned)v.n[0]);
    unsigned zz = fdiv(idx, v.fxy);
    z = (int)zz;
    y = (int)(t - zz * (unsigned)v.n[1]);
}
__device__ __forceinline__ int lv_off(const LView& v, int x, int y, int z) { return x + y * v.sy + z * v.sz; }
// coordinate c + d along an axis of extent n (|d| <= 2, n >= 2): wrapped, or -1 outside
__device__ __forceinline__ int lv_nb(int c, int d, int n, int per) {
    int u = c + d;
    if (per) return u < 0 ? u + n : (u >= n ? u - n : u);
    return (u < 0 || u >= n) ? -1 : u;
}

__device__ __forceinline__ int lv_map(int u, int n, int per) {
    if ((unsigned)u < (unsigned)n) return u;
    if (!per) return -1;
    u += u < 0 ? n : -n;
    if ((unsigned)u < (unsigned)n) return u;
    // a tile past the end of a short periodic axis can reach beyond one period: reduce fully so
    // that every staged read stays on the grid
    const int m = u % n;
    return m < 0 ? m + n : m;
}
// index rule of the restriction along one axis (k_lp_restrict): fine point raw of coarse level c,
// wrapped once by the coarse period on a periodic axis; -1 outside the fine box
__device__ __forceinline__ int rs_map(int raw, const LView& f, const LView& c, int ax) {
    if (f.per[ax]) {
        const int nc2 = 2 * c.n[ax];
        raw = raw < 0 ? raw + nc2 : (raw >= nc2 ? raw - nc2 : raw);
        return raw < f.n[ax] ? raw : -1;
    }
    return (raw >= 0 && raw < f.n[ax]) ? raw : -1;
}

// ------------------------------------------------------------------------------------
// The levels of the hierarchy inside a cooperative launch: restrictions, level operators, and the coarse
// part, levels m .. nlev - 1, down and up again.
//
// As a launch per level and direction, with the coarsest levels in one CTA, the coarse part was a chain of
// latency-bound kernels: 9.7 + 8.0 (restrictions) + 32 (one CTA) + 10.8 + 10.7 us of the 145 us of an
// iteration of 63 x 63 x 256 nodes, the same for grids of any size.  Here a level's voxels are spread over
// all SMs with a grid barrier between levels, and the first level of at most kLpDenseMost voxels takes
// everything below it with it: e = A z with the dense matrix A of op + P (...) R, formed when the weights
// change (lp_build_dense, 2048 columns in about 0.3 ms) and read from L2, 16 MB at most, by one warp per row.
// ------------------------------------------------------------------------------------
constexpr int kLpMidMost = 65536;   // voxels of the first level that joins the coarse launch
constexpr int kLvThr = 512;         // threads of a CTA of the persistent kernels
struct LpCoarseLevels {
    int m, ld, nlev;                 // ld: the dense level (nlev: none)
    LView f0;                        // level m - 1 (its restricted input; the residual if m == 1)
    LView z[kLpMaxLevels], e[kLpMaxLevels];
    const float* fold[kLpMaxLevels];  // folded stencils of a network level, nullptr: diagonal scaling
    float inv_diag[kLpMaxLevels];
    const float* dense;              // rows of `pitch` floats
    int pitch;
};
// the levels from m on of a hierarchy whose level m - 1 is f0
inline void lp_coarse_setup(const LpState& L, int m, const LView& f0, LpCoarseLevels& a) {
    a = LpCoarseLevels{};
    a.nlev = L.nlev;
    a.m = m;
    a.f0 = f0;
    a.ld = std::max(m, L.dense_level);
    for (int l = L.nlev - 1; l >= m; l--) {
        a.z[l] = lp_level_view(L, l, L.z[l]);
        a.e[l] = lp_level_view(L, l, L.e[l]);
        a.fold[l] = l <= kLpNetLevels ? L.fold + (l - 1) * kLpFoldStride : nullptr;
        a.inv_diag[l] = (float)(1.0 / L.diag[l]);
    }
    // a hierarchy whose dense level lies above m (small grids): the level's own matrix is not the dense
    // one, so its levels are applied one by one
    if (a.ld != L.dense_level) a.ld = L.nlev;
    a.dense = L.dense;
    a.pitch = L.dense_pitch;
}

// shared working set of the level functions: the 27 face-class stencils of every network level (class 0:
// the interior one; rows of 125 padded to 128 so that four coefficients are one read), a staged tile
constexpr int kLvTile = 2304;  // the largest halo: 36 x 8 x 8 (or 8 x 8 x 36)
struct LevelSmem {
    LpCoarseLevels lev;  // a copy of the launch's: indexed by level, it is read from here in tens of cycles
    int pad[2];
    float k5[kLpNetLevels][27][128];
    float tile[kLvTile];
    int mx[64], myz[320];  // offsets of a staged tile's points and rows (-1: outside)
};
// The stencils of the face classes that occur (a periodic axis has no faces: 3 of 27 classes with two of
// them), as asynchronous copies: lp_levels_ready waits for the calling thread's
__device__ __forceinline__ void lp_load_levels(LevelSmem& sm, const LpCoarseLevels& lev, int first, int nlev, int nt) {
    if (threadIdx.x == 0) sm.lev = lev;
    const int lane = threadIdx.x & 31;
    for (int l = first; l < nlev && l <= kLpNetLevels; l++)
        for (int cls = threadIdx.x >> 5; cls < 27; cls += nt >> 5) {
            const int* per = lev.z[l].per;
            if ((per[0] && cls % 3) || (per[1] && cls / 3 % 3) || (per[2] && cls / 9)) continue;
            const float* src = lev.fold[l] + kLpFold + 125 * cls;
#pragma unroll
            for (int d = lane; d < 128; d += 32) {
                float* dst = &sm.k5[l - 1][cls][d];
                if (d < 125)
                    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((unsigned)__cvta_generic_to_shared(dst)),
                                 "l"(src + d)
                                 : "memory");
                else
                    *dst = 0.f;
            }
        }
}
__device__ __forceinline__ void lp_levels_ready() { asm volatile("cp.async.wait_all;" ::: "memory"); }
static_assert(kLvTile >= kLpDenseMost, "the dense level's values lie in the staged tile's place");
// a value of a level: shared memory, or global memory that other CTAs write (L2)
template <bool SH>
__device__ __forceinline__ float lp_ld(const float* p) {
    return SH ? *p : __ldcg(p);
}
// z_c = R z_f (index rules of k_lp_restrict): four lanes per coarse voxel, one fine plane each
template <bool SH>
__device__ __forceinline__ void lp_restrict_level(const LView f, const LView c, int cta, int nctas) {
    const float w4[4] = {0.25f, 0.75f, 0.75f, 0.25f};
    const int lane = threadIdx.x & 31;
    // the warps of all CTAs in turn, so that a small level is spread over every SM
    for (int v0 = 8 * ((threadIdx.x >> 5) * nctas + cta); v0 < c.nvox; v0 += 8 * nctas * (kLvThr / 32)) {
        const int v = v0 + (lane >> 2), kz = lane & 3;
        int cc[3];
        lv_decode(c, (unsigned)min(v, c.nvox - 1), cc[0], cc[1], cc[2]);
        const int uz = rs_map(2 * cc[2] + kz - 1, f, c, 2);
        int ox[4], oy[4];
#pragma unroll
        for (int k = 0; k < 4; k++) {
            ox[k] = rs_map(2 * cc[0] + k - 1, f, c, 0);
            const int uy = rs_map(2 * cc[1] + k - 1, f, c, 1);
            oy[k] = uy < 0 ? -1 : uy * f.sy;
        }
        const float* p = f.a + max(uz, 0) * f.sz;
        float a[4][4];
#pragma unroll
        for (int ky = 0; ky < 4; ky++)
#pragma unroll
            for (int kx = 0; kx < 4; kx++)
                a[ky][kx] = (ox[kx] | oy[ky] | uz) >= 0 ? lp_ld<SH>(p + oy[ky] + ox[kx]) : 0.f;
        float acc = 0.f;
#pragma unroll
        for (int ky = 0; ky < 4; ky++)
            acc += w4[ky] * (w4[0] * a[ky][0] + w4[1] * a[ky][1] + w4[2] * a[ky][2] + w4[3] * a[ky][3]);
        acc *= (kz == 0 || kz == 3) ? 0.25f : 0.75f;
        acc += __shfl_xor_sync(0xffffffffu, acc, 1);
        acc += __shfl_xor_sync(0xffffffffu, acc, 2);
        if (kz == 0 && v < c.nvox) c.a[v] = acc;
    }
}
// (P e) at voxel c of the level above e: the eight corners, offsets formed per axis
template <bool SH>
__device__ __forceinline__ float lp_prolong_level(const LView& e, const int (&c)[3]) {
    int o[3][2];
    const int st[3] = {1, e.sy, e.sz};
#pragma unroll
    for (int ax = 0; ax < 3; ax++) {
        const int c0 = c[ax] >> 1, u = lv_nb(c0, (c[ax] & 1) ? 1 : -1, e.n[ax], e.per[ax]);
        o[ax][0] = c0 * st[ax];
        o[ax][1] = u < 0 ? -1 : u * st[ax];
    }
    float v[8];
#pragma unroll
    for (int k = 0; k < 8; k++) {
        const int a = o[0][k & 1], b = o[1][(k >> 1) & 1], d = o[2][k >> 2];
        v[k] = (a | b | d) >= 0 ? lp_ld<SH>(e.a + a + b + d) : 0.f;
    }
    float acc[4];
#pragma unroll
    for (int k = 0; k < 4; k++) acc[k] = 0.75f * v[2 * k] + 0.25f * v[2 * k + 1];
    return 0.75f * (0.75f * acc[0] + 0.25f * acc[1]) + 0.25f * (0.75f * acc[2] + 0.25f * acc[3]);
}
// e_l = op(z) + P e on tiles of kLvThr / TPV voxels of a shape that follows the level's (powers of two),
// TPV threads per voxel: the tile and its two-voxel halo are staged, a thread forms its rows of the 125 taps
// with its face class's stencil.  cta, nctas: the tiles' owners.  All threads of a CTA call it together.
template <bool ZSH, bool ESH, int TPV>
__device__ __forceinline__ void lp_net_tiles(const LView& z, const LView& e, const LView& out, const float (*k5)[128],
                                             LevelSmem& sm, int cta, int nctas) {
    constexpr int kLg = TPV == 1 ? 9 : 7;  // log2 of a tile's voxels
    static_assert((kLvThr / TPV) == 1 << kLg, "the shapes below are for 512 and 128 voxels");
    const int tid = threadIdx.x, vox = tid / TPV, part = tid % TPV;
    // shape: x up to 32 (16 of 128), then y up to 8, the rest in z
    const int lx = min(z.n[0] > 16 ? 5 : (z.n[0] > 8 ? 4 : (z.n[0] > 4 ? 3 : 2)), kLg == 9 ? 5 : 4);
    const int ly = min(z.n[1] > 4 ? 3 : 2, kLg - (kLg == 9 ? 2 : 1) - lx), lz = kLg - lx - ly;
    const int HX = (1 << lx) + 4, HY = (1 << ly) + 4, HZ = (1 << lz) + 4, rows = HY * HZ;
    const int bxn = (z.n[0] + (1 << lx) - 1) >> lx, byn = (z.n[1] + (1 << ly) - 1) >> ly,
              bzn = (z.n[2] + (1 << lz) - 1) >> lz;
    const int tx = vox & ((1 << lx) - 1), ty = (vox >> lx) & ((1 << ly) - 1), tz = vox >> (lx + ly);
    const int lane = tid & 31, wp = tid >> 5;
    for (int tile = cta; tile < bxn * byn * bzn; tile += nctas) {
        const int q = tile / bxn, x0 = (tile - q * bxn) << lx, y0 = (q % byn) << ly, z0 = (q / byn) << lz;
        __syncthreads();  // the tile before has been read
        if (tid < HX) sm.mx[tid] = lv_map(x0 - 2 + tid, z.n[0], z.per[0]);
        for (int r = tid; r < rows; r += kLvThr) {
            const int uy = lv_map(y0 - 2 + r % HY, z.n[1], z.per[1]), uz = lv_map(z0 - 2 + r / HY, z.n[2], z.per[2]);
            sm.myz[r] = (uy | uz) < 0 ? -1 : uy * z.sy + uz * z.sz;
        }
        const int c[3] = {x0 + tx, y0 + ty, z0 + tz};
        const bool live = c[0] < z.n[0] && c[1] < z.n[1] && c[2] < z.n[2];
        __syncthreads();
        // rows wp, wp + 16, ... a lane the points lane and lane + 32 of a row
        const int ox = lane < HX ? sm.mx[lane] : -1, ox2 = lane + 32 < HX ? sm.mx[lane + 32] : -1;
        for (int r0 = wp; r0 < rows; r0 += 4 * (kLvThr / 32)) {
            float v[4], v2[4];
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const int r = r0 + k * (kLvThr / 32);
                const int o = r < rows ? sm.myz[r] : -1;
                v[k] = (o | ox) >= 0 ? lp_ld<ZSH>(z.a + o + ox) : 0.f;
                v2[k] = (o | ox2) >= 0 ? lp_ld<ZSH>(z.a + o + ox2) : 0.f;
            }
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const int r = r0 + k * (kLvThr / 32);
                if (r >= rows) continue;
                if (lane < HX) sm.tile[r * HX + lane] = v[k];
                if (lane + 32 < HX) sm.tile[r * HX + lane + 32] = v2[k];
            }
        }
        const float up = e.a && live && part == 0 ? lp_prolong_level<ESH>(e, c) : 0.f;
        __syncthreads();
        int cls = 0, mul = 1;
#pragma unroll
        for (int ax = 0; ax < 3; ax++) {
            if (!z.per[ax]) cls += mul * (c[ax] == 0 ? 1 : (c[ax] == z.n[ax] - 1 ? 2 : 0));
            mul *= 3;
        }
        const float* p = sm.tile + tx + HX * (ty + HY * tz);
        const float* kk = k5[live ? cls : 0];
        float acc[2] = {up, 0.f};
        if (TPV == 1) {
            const float4* kk4 = reinterpret_cast<const float4*>(kk);
            float4 k4 = kk4[0];
#pragma unroll
            for (int row = 0; row < 25; row++) {
                const float* pr = p + HX * (row % 5 + HY * (row / 5));
#pragma unroll
                for (int dx = 0; dx < 5; dx++) {
                    const int m = 5 * row + dx;
                    if ((m & 3) == 0) k4 = kk4[m >> 2];
                    const float w = (m & 3) == 0 ? k4.x : (m & 3) == 1 ? k4.y : (m & 3) == 2 ? k4.z : k4.w;
                    acc[row & 1] = fmaf(w, pr[dx], acc[row & 1]);
                }
            }
            if (live) out.a[lv_off(out, c[0], c[1], c[2])] = acc[0] + acc[1];
        } else {
#pragma unroll
            for (int q5 = 0; q5 < (25 + TPV - 1) / TPV; q5++) {
                const int row = part + TPV * q5;
                if (row >= 25) break;
                const float* pr = p + HX * (row % 5 + HY * (row / 5));
#pragma unroll
                for (int dx = 0; dx < 5; dx++) acc[q5 & 1] = fmaf(kk[5 * row + dx], pr[dx], acc[q5 & 1]);
            }
            float s = acc[0] + acc[1];
#pragma unroll
            for (int o = 1; o < TPV; o *= 2) s += __shfl_xor_sync(0xffffffffu, s, o);
            if (live && part == 0) out.a[lv_off(out, c[0], c[1], c[2])] = s;
        }
    }
}
// four threads per voxel on levels whose tiles of 512 would leave SMs idle
template <bool ZSH, bool ESH>
__device__ __forceinline__ void lp_net_level(const LView z, const LView e, const LView out, const float (*k5)[128],
                                             LevelSmem& sm, int cta, int nctas) {
    if (out.nvox <= 256 * nctas)
        lp_net_tiles<ZSH, ESH, 4>(z, e, out, k5, sm, cta, nctas);
    else
        lp_net_tiles<ZSH, ESH, 1>(z, e, out, k5, sm, cta, nctas);
}
// e_l = z / diagonal + P e
template <bool ZSH, bool ESH>
__device__ __forceinline__ void lp_diag_level(const LView& z, const LView& e, const LView& out, float inv_diag, int t, int nthr) {
    for (int v = t; v < out.nvox; v += nthr) {
        int c[3];
        lv_decode(out, (unsigned)v, c[0], c[1], c[2]);
        const float zv = lp_ld<ZSH>(z.a + lv_off(z, c[0], c[1], c[2]));
        out.a[v] = inv_diag * zv + (e.a ? lp_prolong_level<ESH>(e, c) : 0.f);
    }
}
template <bool ZSH, bool ESH>
__device__ __forceinline__ void lp_up_level(const LView& z, const LView& e, const LView& out, int l, const float* fold,
                                            float inv_diag, LevelSmem& sm, int cta, int nctas) {
    if (fold)
        lp_net_level<ZSH, ESH>(z, e, out, sm.k5[min(l, kLpNetLevels) - 1], sm, cta, nctas);
    else
        lp_diag_level<ZSH, ESH>(z, e, out, inv_diag, cta * kLvThr + (int)threadIdx.x, nctas * kLvThr);
}
// e = A z of the dense level: z in shared memory (pitch floats, zero-padded), one warp per row
__device__ __forceinline__ void lp_dense_level(const LpCoarseLevels& a, float* zs) {
    const int tid = threadIdx.x, lane = tid & 31, n = a.z[a.ld].nvox, n4 = a.pitch >> 2;
    const float* z = a.z[a.ld].a;
    float* e = a.e[a.ld].a;
    __syncthreads();
    for (int x = tid; x < a.pitch; x += kLvThr) zs[x] = x < n ? __ldcg(z + x) : 0.f;
    __syncthreads();
    const float4* z4 = reinterpret_cast<const float4*>(zs);
    for (int row = (tid >> 5) * gridDim.x + blockIdx.x; row < n; row += gridDim.x * (kLvThr / 32)) {
        const float4* A = reinterpret_cast<const float4*>(a.dense + (size_t)row * a.pitch);
        float acc[4] = {0.f, 0.f, 0.f, 0.f};
        for (int q0 = lane; q0 < n4; q0 += 32 * 8) {
            float4 v[8];  // eight rows of lanes in flight
#pragma unroll
            for (int k = 0; k < 8; k++) v[k] = q0 + 32 * k < n4 ? __ldg(A + q0 + 32 * k) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int k = 0; k < 8; k++) {
                if (q0 + 32 * k >= n4) break;
                const float4 y = z4[q0 + 32 * k];
                acc[0] = fmaf(v[k].x, y.x, acc[0]);
                acc[1] = fmaf(v[k].y, y.y, acc[1]);
                acc[2] = fmaf(v[k].z, y.z, acc[2]);
                acc[3] = fmaf(v[k].w, y.w, acc[3]);
            }
        }
        float s = (acc[0] + acc[1]) + (acc[2] + acc[3]);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (lane == 0) e[row] = s;
    }
}
// z of levels m .. and e of levels .. m from f0's values (published before the call; e of level m is
// published by the caller's next barrier).  False when a grid barrier ran out.  LOADING: lp_load_levels may
// still be on its way.
template <bool LOADING>
__device__ __forceinline__ bool lp_coarse_levels(const LpCoarseLevels& a, LevelSmem& sm, const GridWait& wait,
                                                 unsigned& target, int* s_fail) {
    const int cta = blockIdx.x, nctas = gridDim.x;
    const int last = min(a.ld, a.nlev - 1);  // the last level that is restricted
    bool ok = true;
    for (int l = a.m; l <= last && ok; l++) {
        lp_restrict_level<false>(l == a.m ? a.f0 : a.z[l - 1], a.z[l], cta, nctas);
        if (l == last && LOADING) lp_levels_ready();  // published to the CTA by the barrier
        ok = grid_barrier(wait, target, s_fail);
    }
    for (int l = last; l >= a.m && ok; l--) {
        if (l == a.ld) {
            lp_dense_level(a, sm.tile);
        } else {
            LView up{};
            if (l + 1 < a.nlev) up = a.e[l + 1];
            lp_up_level<false, false>(a.z[l], up, a.e[l], l, a.fold[l], a.inv_diag[l], sm, cta, nctas);
        }
        if (l > a.m) ok = grid_barrier(wait, target, s_fail);
    }
    return ok;
}

}  // namespace pic
