// Poisson inner solvers as one persistent kernel over the whole GPU, for grids beyond one cluster
// (pic_cluster.cu) whose inner state fits the shared memory of all SMs together (up to 2.3 million nodes of
// the CG, 2.7 million of the sweeps): SOR sweeps and the Jacobi-preconditioned flexible CG of L e = r.
//
// As separate launches an iteration of 129^3 nodes reads and writes its six arrays through L2 twice
// (52 us), and one of a few 100 000 nodes is mostly launch and drain.  Here one cooperative launch runs
// a batch of sweeps or the whole inner CG solve.  Every CTA owns a contiguous range of nodes and keeps
// their unknowns in shared memory and registers; only the direction (or the SOR iterate) is also written
// to global memory, where the CTAs that own its neighbours read it through L2.  Passes are separated by
// grid barriers: one arrival counter and a bounded poll by one thread, 1.5 us on 152 CTAs with the
// publication of the writes before it.  (Measured beside it: a flag per CTA that only the neighbours poll
// 1.5 us at best and 4 us with the flags in one cache line; all CTAs polling all partial sums 2.3 us.)
//
// Measured: 25 sweeps of 65 x 65 x 97 nodes 168 us (325 us as 50 launches); a CG iteration of 65 x 65 x 97
// nodes 8.1 us, of 129^3 nodes 14.7 us (52 us as two launches), of which the three barriers and sums are 6 us.
//
// The arithmetic of a node is that of k_rbsor and k_pcg_* (pic_fields.cu), in the same order; sums: grid_total.
#include <algorithm>
#include "pic_ff.cuh"
#include "pic_grid_sync.cuh"
#include "pic_stencil.cuh"

namespace pic {
namespace {

constexpr int kThr = 1024;     // threads of the sweeps
constexpr int kPcgThr = 512;   // threads of the CG: 128 registers hold a group's neighbour rows
constexpr size_t kSmemMost = 216 * 1024;   // dynamic shared memory of a CTA

// flags of a node: FREE (1), mirror mask (6 bits), wraps (6 bits: at the low / high end of a periodic
// axis x, y, z); 0 for a node without an unknown
__device__ __forceinline__ unsigned node_flags(const GridDev& g, int n, unsigned kd) {
    if ((kd & 3) != kFree) return 0u;
    int i, j, k;
    node_ijk(g, n, i, j, k);
    unsigned f = 1u | ((kd >> 2) & 63u) << 1;
    if (g.periodic[0]) f |= (i == 0 ? 1u << 7 : 0u) | (i == g.ni - 2 ? 1u << 8 : 0u);
    if (g.periodic[1]) f |= (j == 0 ? 1u << 9 : 0u) | (j == g.nj - 2 ? 1u << 10 : 0u);
    if (g.periodic[2]) f |= (k == 0 ? 1u << 11 : 0u) | (k == g.nk - 2 ? 1u << 12 : 0u);
    return f;
}
// index offsets of the six neighbours of a node
__device__ __forceinline__ void neighbour_offsets(const GridDev& g, unsigned f, int (&o)[6]) {
    const int nij = g.ni * g.nj;
    o[0] = (f & (1u << 7)) ? g.ni - 2 : -1;
    o[1] = (f & (1u << 8)) ? 2 - g.ni : 1;
    o[2] = (f & (1u << 9)) ? (g.nj - 2) * g.ni : -g.ni;
    o[3] = (f & (1u << 10)) ? (2 - g.nj) * g.ni : g.ni;
    o[4] = (f & (1u << 11)) ? (g.nk - 2) * nij : -nij;
    o[5] = (f & (1u << 12)) ? (2 - g.nk) * nij : nij;
}
// off-diagonal sum of a node at local index l: neighbours of the CTA's own range from shared memory,
// the others from global memory (L2: other CTAs write them); zero on MIRROR and FIXED nodes
__device__ __forceinline__ float off_sum(const GridDev& g, const float (&c3)[3], const float* A, const float* G, int l,
                                         int len, unsigned f) {
    int o[6];
    neighbour_offsets(g, f, o);
    float v[6];
#pragma unroll
    for (int d = 0; d < 6; d++) {
        const int q = l + o[d];
        v[d] = (unsigned)q < (unsigned)len ? A[q] : __ldcg(G + q);
    }
    float off = 0.f;
#pragma unroll
    for (int d = 0; d < 6; d++) off += c3[d >> 1] * v[d];
    return off;
}
__device__ __forceinline__ void diag_table(const GridDev& g, float (&c3)[3], float* dia) {
    for (int d = 0; d < 3; d++) c3[d] = g.inv_dx[d] * g.inv_dx[d];
    if (threadIdx.x < 64) {
        float dg = 0.f;
        for (int d = 0; d < 6; d++)
            if (!(threadIdx.x & (1u << d))) dg += c3[d >> 1];
        dia[threadIdx.x] = dg;
    }
}

// ------------------------------------------------------------------------------------
// SOR sweeps (passes as in k_sor_cluster: the two colours, then the nodes on the seams of odd periodic
// axes by number of seams and colour, relaxed with omega = 1); e from zero
// ------------------------------------------------------------------------------------
__global__ void __launch_bounds__(kThr, 1) k_sor_grid(GridDev g, float* __restrict__ e, const float* __restrict__ r,
                                                      const uint16_t* __restrict__ kind, float omega, int sweeps,
                                                      int chunk, GridWait wait) {
    extern __shared__ __align__(16) float sm[];
    uint2* L = reinterpret_cast<uint2*>(sm);  // chunk entries by pass: local index (16 bits), flags; r
    float* E = sm + 2 * (size_t)chunk;
    __shared__ int cnt[8], start[9], s_fail;
    __shared__ float dia[64];
    const int tid = threadIdx.x, n0 = blockIdx.x * chunk, len = min(chunk, g.nv - n0);
    float c3[3];
    diag_table(g, c3, dia);
    if (tid < 8) cnt[tid] = 0;
    if (tid == 0) s_fail = 0;
    const bool sx = g.periodic[0] && ((g.ni - 1) & 1), sy = g.periodic[1] && ((g.nj - 1) & 1),
               sz = g.periodic[2] && ((g.nk - 1) & 1);
    const int npass = 2 + 2 * ((int)sx + (int)sy + (int)sz);
    __syncthreads();
    auto pass_of = [&](int n) -> int {
        int i, j, k;
        node_ijk(g, n, i, j, k);
        const int m = (int)(sx && i == g.ni - 2) + (int)(sy && j == g.nj - 2) + (int)(sz && k == g.nk - 2);
        return 2 * m + ((i + j + k) & 1);
    };
    for (int x = tid; x < len; x += kThr) {
        E[x] = 0.f;
        e[n0 + x] = 0.f;
        if ((kind[n0 + x] & 3) == kFree) atomicAdd(&cnt[pass_of(n0 + x)], 1);
    }
    __syncthreads();
    if (tid == 0) {
        start[0] = 0;
        for (int p = 0; p < 8; p++) {
            start[p + 1] = start[p] + cnt[p];
            cnt[p] = start[p];
        }
    }
    __syncthreads();
    for (int x = tid; x < len; x += kThr) {
        const unsigned f = node_flags(g, n0 + x, kind[n0 + x]);
        if (f) L[atomicAdd(&cnt[pass_of(n0 + x)], 1)] = make_uint2((unsigned)x | f << 16, __float_as_uint(r[n0 + x]));
    }
    unsigned target = 0;
    bool ok = grid_barrier(wait, target, &s_fail);  // every e is zero
    float* G = e + n0;
    for (int it = 0; it < sweeps && ok; it++)
        for (int p = 0; p < npass && ok; p++) {
            const float om = p < 2 ? omega : 1.0f;
            for (int y = start[p] + tid; y < start[p + 1]; y += kThr) {
                const uint2 u = L[y];
                const int l = (int)(u.x & 0xFFFFu);
                const unsigned f = u.x >> 16;
                const float off = off_sum(g, c3, E, G, l, len, f);
                const float en = E[l];
                const float v = en + om * ((__uint_as_float(u.y) + off) / dia[(f >> 1) & 63u] - en);
                E[l] = v;
                G[l] = v;
            }
            ok = grid_barrier(wait, target, &s_fail);
        }
    if (!ok && tid == 0) {
        set_error(wait.err, kErrBarrierTimeout);
        *wait.fail = 1;
    }
}

// ------------------------------------------------------------------------------------
// the whole inner CG solve of L e = r from e = 0 (the iteration of k_pcg_k1 / k_pcg_k2)
// ------------------------------------------------------------------------------------
// flag[0]: converged (r.r <= target), flag[1]: iterations done.  A thread owns the groups of four
// consecutive nodes tid + m kPcgThr (m < K) of its CTA's range: d, r and e of a group are one 16-byte word of
// shared memory each, q stays in registers.  What bounds a pass is the latency of the L2 reads of other
// CTAs' nodes, so a group reads its four neighbour rows as aligned 16-byte words that are all in flight
// before one is used (node by node, or row by row, an iteration of 129^3 nodes took 21 us); only groups
// at the ends of a periodic axis, and the first and last of the grid, look up their neighbours one by one.
constexpr unsigned long long kPlain4 = 0x0001000100010001ull, kWrap4 = 0x1F801F801F801F80ull;
template <int K>
__global__ void __launch_bounds__(kPcgThr, 1) k_pcg_grid(GridDev g, float* __restrict__ e, const float* __restrict__ r,
                                                      float* dg, const uint16_t* __restrict__ kind, SumScales sc,
                                                      FF target_rr, int cap, int chunk, int* flag, GridSync* sync,
                                                      GridWait wait) {
    const float sc1[1] = {sc.rz}, sc3[3] = {sc.rz, sc.rz, sc.rr};
    constexpr int kRun = kFp32Nodes / 4;  // groups that a thread adds in FP32
    static_assert(K <= 2 * kRun, "two such sums at most");
    extern __shared__ __align__(16) float sm[];
    float4* D4 = reinterpret_cast<float4*>(sm);
    float4* R4 = D4 + chunk / 4;
    float4* X4 = R4 + chunk / 4;
    unsigned long long* M4 = reinterpret_cast<unsigned long long*>(X4 + chunk / 4);  // four 16-bit flag words
    float* D = sm;
    __shared__ float dia[64], inv[64], s_alpha, s_beta;
    __shared__ float2 wsum[3][kPcgThr / 32];
    __shared__ int s_fail, s_stop;  // s_stop: 1 converged, 3 not a number
    const int tid = threadIdx.x, n0 = blockIdx.x * chunk, len = min(chunk, g.nv - n0);
    const int ng = chunk / 4, nij = g.ni * g.nj;
    float c3[3];
    diag_table(g, c3, dia);
    __syncthreads();
    if (tid < 64) inv[tid] = 1.f / dia[tid];
    if (tid == 0) {
        s_beta = 0.f;
        s_stop = s_fail = 0;
    }
    __syncthreads();
    float* G = dg + n0;
    FF f3[3] = {FF{0.f, 0.f}, FF{0.f, 0.f}, FF{0.f, 0.f}};
    for (int q = tid; q < ng; q += kPcgThr) {
        float rv[4], f = 0.f;
        unsigned long long mm = 0;
#pragma unroll
        for (int c = 0; c < 4; c++) {
            const int x = 4 * q + c;
            const unsigned fl = x < len ? node_flags(g, n0 + x, kind[n0 + x]) : 0u;
            rv[c] = fl ? r[n0 + x] : 0.f;
            if (x < len) G[x] = 0.f;
            mm |= (unsigned long long)fl << (16 * c);
            f += rv[c] * (rv[c] * inv[(fl >> 1) & 63u]);
        }
        f3[0] = ff_acc(f3[0], f);
        D4[q] = X4[q] = make_float4(0.f, 0.f, 0.f, 0.f);
        R4[q] = make_float4(rv[0], rv[1], rv[2], rv[3]);
        M4[q] = mm;
    }
    float2(*part1)[kMostCtas] = sync->part;
    float2(*part3)[kMostCtas] = sync->part + 1;
    unsigned target = 0;
    FF t1[1], t3[3];
    grid_total<3, kPcgThr>(f3, sc3, wsum, part3, wait, target, &s_fail, t3);  // r.z
    FF rz = t3[0];
    const float inv0 = inv[0], dia0 = dia[0];
    __syncthreads();
    int it = 0;
    float Q[K][4];
    while (it < cap && !s_fail) {
        // d = z + beta d (z = r / diagonal; both zero off the unknowns)
        const float beta = s_beta;
#pragma unroll
        for (int m = 0; m < K; m++) {
            const int q = tid + m * kPcgThr;
            if (q >= ng) break;
            const unsigned long long mm = M4[q];
            if (!mm) continue;
            const float4 rv = R4[q], dv = D4[q];
            float4 v;
            if (mm == kPlain4) {
                v = make_float4(rv.x * inv0 + beta * dv.x, rv.y * inv0 + beta * dv.y, rv.z * inv0 + beta * dv.z,
                                rv.w * inv0 + beta * dv.w);
            } else {
                const float a[4] = {rv.x, rv.y, rv.z, rv.w}, b[4] = {dv.x, dv.y, dv.z, dv.w};
                float o[4];
#pragma unroll
                for (int c = 0; c < 4; c++) o[c] = a[c] * inv[(unsigned)(mm >> (16 * c + 1)) & 63u] + beta * b[c];
                v = make_float4(o[0], o[1], o[2], o[3]);
            }
            D4[q] = v;
            if (4 * q + 4 <= len)
                reinterpret_cast<float4*>(G)[q] = v;
            else {  // the grid's last nodes
                const float o[4] = {v.x, v.y, v.z, v.w};
                for (int c = 0; 4 * q + c < len; c++) G[4 * q + c] = o[c];
            }
        }
        if (!grid_barrier(wait, target, &s_fail)) break;
        // q = L d, d.q
        FF v1[1] = {FF{0.f, 0.f}};
        float f1 = 0.f;
#pragma unroll
        for (int m = 0; m < K; m++) {
            const int q = tid + m * kPcgThr;
            Q[m][0] = Q[m][1] = Q[m][2] = Q[m][3] = 0.f;
            if (q >= ng) break;
            if (m == kRun) {
                v1[0].hi = f1;
                f1 = 0.f;
            }
            const unsigned long long mm = M4[q];
            if (!mm) continue;
            const int l = 4 * q;
            const float4 d4 = D4[q];
            float nb[4][6];  // neighbours of the four nodes (zero on MIRROR and FIXED nodes)
            if (!(mm & kWrap4) && n0 + l - nij - 3 >= 0 && n0 + l + nij + 8 <= g.nv) {
                // rows at a fixed distance: two 16-byte words each, all in flight at once
                const float xm = l > 0 ? D[l - 1] : __ldcg(G + l - 1);
                const float xp = l + 4 < len ? D[l + 4] : __ldcg(G + l + 4);
                const int at[4] = {l - g.ni, l + g.ni, l - nij, l + nij};
                float4 A[4], B[4];
#pragma unroll
                for (int t = 0; t < 4; t++) {
                    const int o = at[t] & ~3;
                    const bool own = o >= 0 && o + 8 <= chunk;
                    A[t] = own ? D4[o >> 2] : __ldcg(reinterpret_cast<const float4*>(G + o));
                    B[t] = own ? D4[(o >> 2) + 1] : __ldcg(reinterpret_cast<const float4*>(G + o) + 1);
                }
                const float dv[6] = {xm, d4.x, d4.y, d4.z, d4.w, xp};
#pragma unroll
                for (int c = 0; c < 4; c++) {
                    nb[c][0] = dv[c];
                    nb[c][1] = dv[c + 2];
                }
#pragma unroll
                for (int t = 0; t < 4; t++) {
                    const int sh = at[t] & 3;  // the same for every group
                    const float w[8] = {A[t].x, A[t].y, A[t].z, A[t].w, B[t].x, B[t].y, B[t].z, B[t].w};
                    float h[6];
#pragma unroll
                    for (int c = 0; c < 5; c++) h[c] = (sh & 2) ? w[c + 2] : w[c];
#pragma unroll
                    for (int c = 0; c < 4; c++) nb[c][2 + t] = (sh & 1) ? h[c + 1] : h[c];
                }
            } else {
#pragma unroll
                for (int c = 0; c < 4; c++) {
                    const unsigned f = (unsigned)(mm >> (16 * c)) & 0xFFFFu;
                    int o[6];
                    neighbour_offsets(g, f, o);
#pragma unroll
                    for (int d = 0; d < 6; d++) {
                        const int y = l + c + o[d];
                        nb[c][d] = !f ? 0.f : ((unsigned)y < (unsigned)len ? D[y] : __ldcg(G + y));
                    }
                }
            }
            const float dv[4] = {d4.x, d4.y, d4.z, d4.w};
#pragma unroll
            for (int c = 0; c < 4; c++) {
                const unsigned f = (unsigned)(mm >> (16 * c)) & 0xFFFFu;
                float off = 0.f;
#pragma unroll
                for (int d = 0; d < 6; d++) off += c3[d >> 1] * nb[c][d];
                const float di = mm == kPlain4 ? dia0 : dia[(f >> 1) & 63u];
                Q[m][c] = f ? di * dv[c] - off : 0.f;
                f1 += dv[c] * Q[m][c];
            }
        }
        v1[0] = ff_acc(v1[0], f1);
        grid_total<1, kPcgThr>(v1, sc1, wsum, part1, wait, target, &s_fail, t1);
        if (tid == 0) s_alpha = t1[0].hi != 0.f ? ff_ratio(rz, t1[0]) : 0.f;
        __syncthreads();
        if (s_fail) break;
        // e += alpha d, r -= alpha q, z = r / diagonal
        const float alpha = s_alpha;
        FF v3[3] = {FF{0.f, 0.f}, FF{0.f, 0.f}, FF{0.f, 0.f}};
        float f[3] = {0.f, 0.f, 0.f};
#pragma unroll
        for (int m = 0; m < K; m++) {
            const int q = tid + m * kPcgThr;
            if (q >= ng) break;
            if (m == kRun)
#pragma unroll
                for (int c = 0; c < 3; c++) {
                    v3[c].hi = f[c];
                    f[c] = 0.f;
                }
            const unsigned long long mm = M4[q];
            if (!mm) continue;
            const float4 d4 = D4[q], x4 = X4[q], r4 = R4[q];
            const float dv[4] = {d4.x, d4.y, d4.z, d4.w}, rv[4] = {r4.x, r4.y, r4.z, r4.w};
            float xv[4] = {x4.x, x4.y, x4.z, x4.w}, rn[4];
#pragma unroll
            for (int c = 0; c < 4; c++) {  // d and q are zero off the unknowns, and so is r
                const float iv = mm == kPlain4 ? inv0 : inv[(unsigned)(mm >> (16 * c + 1)) & 63u];
                xv[c] += alpha * dv[c];
                rn[c] = rv[c] - alpha * Q[m][c];
                f[0] += rn[c] * (rn[c] * iv);
                f[1] += rn[c] * (rv[c] * iv);
                f[2] += rn[c] * rn[c];
            }
            X4[q] = make_float4(xv[0], xv[1], xv[2], xv[3]);
            R4[q] = make_float4(rn[0], rn[1], rn[2], rn[3]);
        }
#pragma unroll
        for (int c = 0; c < 3; c++) v3[c] = ff_acc(v3[c], f[c]);
        grid_total<3, kPcgThr>(v3, sc3, wsum, part3, wait, target, &s_fail, t3);
        it++;
        if (tid == 0) {
            const float over = (t3[2].hi - target_rr.hi) + (t3[2].lo - target_rr.lo);
            if (!(over > 0.f)) s_stop = over <= 0.f ? 1 : 3;
            s_beta = ff_ratio(ff_add(t3[0], ff_neg(t3[1])), rz);
        }
        rz = t3[0];
        __syncthreads();
        if (s_stop) break;
    }
    if (tid == 0) {
        if (blockIdx.x == 0) {
            flag[0] = !s_fail && s_stop == 1;
            flag[1] = it;
        }
        if (s_fail) {
            set_error(wait.err, kErrBarrierTimeout);
            *wait.fail = 1;
        }
    }
    for (int x = tid; x < len; x += kPcgThr) e[n0 + x] = reinterpret_cast<const float*>(X4)[x];
}

// nodes per CTA over the GPU's SMs (whole warps), and the CTAs that takes
int chunk_of(const GridDev& g, int sms) { return ((g.nv + sms - 1) / sms + 31) / 32 * 32; }
size_t sor_bytes(int chunk) { return 12 * (size_t)chunk; }
size_t pcg_bytes(int chunk) { return 14 * (size_t)chunk; }
using PcgKernel = void (*)(GridDev, float*, const float*, float*, const uint16_t*, SumScales, FF, int, int, int*, GridSync*,
                           GridWait);
PcgKernel pcg_kernel(int chunk) {
    if (chunk <= 4 * kPcgThr) return k_pcg_grid<1>;
    if (chunk <= 8 * kPcgThr) return k_pcg_grid<2>;
    if (chunk <= 16 * kPcgThr) return k_pcg_grid<4>;
    if (chunk <= 32 * kPcgThr) return k_pcg_grid<8>;
    return nullptr;
}
template <class K>
bool fits(K kernel, int threads, size_t bytes) {
    cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemMost);
    int n = 0;
    const bool ok = bytes <= kSmemMost &&
                    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, threads, bytes) == cudaSuccess && n > 0;
    if (!ok) cudaGetLastError();
    return ok;
}
}  // namespace

int plan_sor_grid(const GridDev& g, int sms) {
    const int c = chunk_of(g, sms);
    return sms <= kMostCtas && c <= 65535 && fits(k_sor_grid, kThr, sor_bytes(c)) ? c : 0;
}
int plan_pcg_grid(const GridDev& g, int sms) {
    const int c = chunk_of(g, sms);
    const PcgKernel k = pcg_kernel(c);
    return sms <= kMostCtas && k && fits(k, kPcgThr, pcg_bytes(c)) ? c : 0;
}

void launch_sor_grid(const GridDev& g, SolveWork& w, float omega, int sweeps, int chunk, cudaStream_t s) {
    const uint16_t* kd = reinterpret_cast<const uint16_t*>(w.kind);
    const float* r = w.r;
    GridDev gg = g;
    GridSync* sync = reinterpret_cast<GridSync*>(w.gpart);
    GridWait gw{&sync->arrived, w.wait_polls, w.err, w.flag + 2};
    cudaMemsetAsync(sync, 0, sizeof(unsigned), s);
    void* args[] = {&gg, &w.e, &r, &kd, &omega, &sweeps, &chunk, &gw};
    cudaLaunchCooperativeKernel((const void*)k_sor_grid, dim3((g.nv + chunk - 1) / chunk), dim3(kThr), args,
                                sor_bytes(chunk), s);
}
void launch_pcg_grid(const GridDev& g, SolveWork& w, double r2, double target_rr, int cap, int chunk, cudaStream_t s) {
    const uint16_t* kd = reinterpret_cast<const uint16_t*>(w.kind);
    const float* r = w.r;
    GridDev gg = g;
    // the shared state lies in the node kernels' partial-sum buffer (kParts x 8 doubles at least)
    static_assert(sizeof(GridSync) <= sizeof(double) * 8 * kParts, "the partial-sum buffer holds the grid's state");
    GridSync* sync = reinterpret_cast<GridSync*>(w.gpart);
    GridWait gw{&sync->arrived, w.wait_polls, w.err, w.flag + 2};
    cudaMemsetAsync(sync, 0, sizeof(unsigned), s);
    SumScales sc = sum_scales(g, r2);
    FF t = ff_from_double(target_rr * sc.rr);
    void* args[] = {&gg, &w.e, &r, &w.d, &kd, &sc, &t, &cap, &chunk, &w.flag, &sync, &gw};
    cudaLaunchCooperativeKernel((const void*)pcg_kernel(chunk), dim3((g.nv + chunk - 1) / chunk), dim3(kPcgThr), args,
                                pcg_bytes(chunk), s);
}

}  // namespace pic
