// Poisson inner solvers on one thread-block cluster, for grids whose inner state fits the shared
// memory of up to 16 SMs: SOR sweeps and the Jacobi-preconditioned flexible CG of L e = r.
//
// On such grids (the reference's own sizes: 21^3, 31 x 31 x 51 nodes) a sweep or an iteration is a few
// microseconds of work, and two launches each, with a grid-wide sum and a host check in between, cost
// ten times that.  Here one launch runs all sweeps of a batch, or the whole inner CG solve: the planes
// of the grid are split over the CTAs of a cluster, every CTA keeps its planes in shared memory, and
// the two boundary planes go into the neighbours' halo planes through distributed shared memory as
// they are computed (st.async: the data and its completion on the receiver's mbarrier in one message, so
// a CTA waits for its neighbours' planes only, never for a cluster-wide barrier).  Every wait is bounded; a CTA
// whose wait runs out leaves its loop and joins the others at the closing cluster barrier, so that no CTA's
// shared memory goes away under a message.
//
// Measured: 25 sweeps of 21^3 nodes 34 us on 16 CTAs (60 on 4, 112 on 1; about 190 as 50 launches), of
// 31 x 31 x 51 nodes 71 us; a CG iteration of 21^3 nodes 2.8 us, of 31 x 31 x 51 nodes 4.6 us (21 us as two
// launches).  More CTAs are faster at every size, so the cluster is as large as the GPU allows.
//
// The arithmetic of a node is that of k_rbsor and k_pcg_* (pic_fields.cu), in the same order.
#include <algorithm>
#include "pic_ff.cuh"
#include "pic_grid_sync.cuh"
#include "pic_stencil.cuh"

namespace pic {
namespace {

// ------------------------------------------------------------------------------------
// cluster primitives
// ------------------------------------------------------------------------------------
__device__ __forceinline__ unsigned cluster_rank() {
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// address of a shared-memory object of this CTA in the CTA of a given rank
__device__ __forceinline__ unsigned map_rank(const void* p, unsigned rank) {
    unsigned a = (unsigned)__cvta_generic_to_shared(p), r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
    return r;
}
// remote stores that count their bytes on an mbarrier of the receiving CTA
__device__ __forceinline__ void st_async2(unsigned a, float x, float y, unsigned bar) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v2.f32 [%0], {%1, %2}, [%3];" ::"r"(a), "f"(x),
                 "f"(y), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void st_async(unsigned a, float v, unsigned bar) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.f32 [%0], %1, [%2];" ::"r"(a), "f"(v), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void bar_init(unsigned long long* bar) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"((unsigned)__cvta_generic_to_shared(bar)) : "memory");
}
__device__ __forceinline__ void bar_expect(unsigned long long* bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"((unsigned)__cvta_generic_to_shared(bar)),
                 "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ bool bar_poll(unsigned long long* bar, unsigned parity, long long limit) {
    const unsigned a = (unsigned)__cvta_generic_to_shared(bar);
    for (long long it = 0; it < limit; it++) {
        unsigned ok;
        asm volatile(
            "{\n .reg .pred p;\n mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
            " selp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(ok)
            : "r"(a), "r"(parity)
            : "memory");
        if (ok) return true;
    }
    return false;
}

// bounded wait; when it runs out, the messages still on their way get the full limit to land
__device__ __forceinline__ bool bar_wait(unsigned long long* bar, unsigned parity, long long limit) {
    if (bar_poll(bar, parity, limit)) return true;
    bar_poll(bar, parity, kMbarWaitPolls);
    return false;
}
// end of a kernel: no CTA leaves while another may still send to it (after a wait that ran out, with
// time for messages that nobody waits for any more)
__device__ __forceinline__ void cluster_leave(bool failed) {
    cluster_sync();
    if (failed)
        for (int q = 0; q < 100; q++) __nanosleep(1000);
    cluster_sync();
}

constexpr int kMaxCtas = 16;

// diagonal of the reduced operator from a mirror mask (direction order -x +x -y +y -z +z)
__device__ __forceinline__ float mask_diag(const float (&c3)[3], unsigned mask) {
    float dg = 0.f;
#pragma unroll
    for (int d = 0; d < 6; d++)
        if (!(mask & (1u << d))) dg += c3[d >> 1];
    return dg;
}

// bound of a wait and where a wait that ran out is recorded
struct ClusterWait {
    long long polls;
    unsigned* err;
    int* fail;
};

// the slab of planes of one CTA, shared by both solvers
struct Slab {
    int nz;      // planes on the ring or stack (a periodic z axis: without the copy plane nk - 1)
    int planes;  // planes per CTA (the last one may own fewer)
    int k0, np;  // this CTA's planes k0 .. k0 + np - 1
    int nij;
    bool has_lo, has_hi;  // a neighbour below, above
    unsigned lo, hi;      // where the first and the last plane's values go there
    unsigned lo_rank, hi_rank;
};
// halo'd array A: plane l of the CTA at A + (l + 1) * nij, the neighbours' planes at 0 and np + 1
__device__ __forceinline__ Slab make_slab(const GridDev& g, int planes, const float* A) {
    Slab s;
    s.nz = g.periodic[2] ? g.nk - 1 : g.nk;
    s.planes = planes;
    s.nij = g.ni * g.nj;
    const int ctas = (s.nz + planes - 1) / planes, rank = (int)cluster_rank();
    s.k0 = rank * planes;
    s.np = min(planes, s.nz - s.k0);
    s.lo = s.hi = s.lo_rank = s.hi_rank = 0;
    s.has_lo = rank > 0 || g.periodic[2];
    s.has_hi = rank < ctas - 1 || g.periodic[2];
    if (s.has_lo) {
        const int prev = rank > 0 ? rank - 1 : ctas - 1;
        const int pnp = min(planes, s.nz - prev * planes);
        s.lo_rank = (unsigned)prev;
        s.lo = map_rank(A + (size_t)(pnp + 1) * s.nij, s.lo_rank);
    }
    if (s.has_hi) {
        s.hi_rank = (unsigned)(rank < ctas - 1 ? rank + 1 : 0);
        s.hi = map_rank(A, s.hi_rank);
    }
    return s;
}
// value v at slot idx of A (own planes): also into the neighbours' halo planes, counted on their barrier
// b (lo_bar, hi_bar: its address there)
__device__ __forceinline__ void put(const Slab& s, float* A, int idx, float v, unsigned lo_bar, unsigned hi_bar) {
    A[idx] = v;
    if (idx < 2 * s.nij && s.has_lo) st_async(s.lo + 4u * (unsigned)(idx - s.nij), v, lo_bar);
    if (idx >= s.np * s.nij && s.has_hi) st_async(s.hi + 4u * (unsigned)(idx - s.np * s.nij), v, hi_bar);
}
// node x of the two halo planes (0 .. 2 nij): its index in the grid, -1 without a neighbour there
__device__ __forceinline__ int halo_node(const Slab& s, int x) {
    const bool up = x >= s.nij;
    if (up ? !s.has_hi : !s.has_lo) return -1;
    int k = up ? s.k0 + s.np : s.k0 - 1;
    k = k < 0 ? s.nz - 1 : (k >= s.nz ? 0 : k);
    return k * s.nij + (up ? x - s.nij : x);
}
// offsets of the in-plane neighbours of a node from its wrap flags (1: i = 0, 2: i = ni - 2, 4: j = 0,
// 8: j = nj - 2, on periodic axes)
__device__ __forceinline__ void plane_nb(const GridDev& g, unsigned wrap, int& xm, int& xp, int& ym, int& yp) {
    xm = (wrap & 1u) ? g.ni - 2 : -1;
    xp = (wrap & 2u) ? 2 - g.ni : 1;
    ym = (wrap & 4u) ? (g.nj - 2) * g.ni : -g.ni;
    yp = (wrap & 8u) ? (2 - g.nj) * g.ni : g.ni;
}
__device__ __forceinline__ unsigned wrap_flags(const GridDev& g, int i, int j) {
    unsigned f = 0;
    if (g.periodic[0]) f |= (i == 0 ? 1u : 0u) | (i == g.ni - 2 ? 2u : 0u);
    if (g.periodic[1]) f |= (j == 0 ? 4u : 0u) | (j == g.nj - 2 ? 8u : 0u);
    return f;
}

// ------------------------------------------------------------------------------------
// SOR sweeps: e from zero, red then black nodes, then the nodes of a seam (a periodic axis with an odd
// number of distinct nodes closes an odd cycle, so its last distinct plane is left out of the two
// colours and relaxed with omega = 1): nodes on one seam by colour, then those on two, then on three,
// so that no two neighbours are updated at once and the result does not depend on timing.
// Every CTA lists its nodes by pass once; a pass is one shared-memory update per listed node, and ends
// when the neighbours' values of the pass have arrived.  The barriers alternate between passes, so no CTA may
// be two passes ahead of a neighbour.  Values bound the drift: a CTA that has all of a neighbour's values of
// pass p knows that the neighbour has left pass p - 1 and done its reads of the halo for p.  A CTA
// without unknowns of a pass in its boundary plane (a wall or a plate there, or a pass that only relaxes a
// seam elsewhere) has no values to send; it sends the neighbour one word that nobody reads instead, as
// it begins the pass.
// ------------------------------------------------------------------------------------
// A list entry is the node's slot (20 bits), mirror mask (6) and wrap flags (4), and its r.  The
// off-diagonal sum needs no mask: e stays zero on MIRROR and FIXED nodes.
__global__ void __launch_bounds__(1024, 1) k_sor_cluster(GridDev g, float* __restrict__ e, const float* __restrict__ r,
                                                         const uint16_t* __restrict__ kind, float omega, int sweeps,
                                                         int planes, ClusterWait wait) {
    extern __shared__ __align__(16) float sm[];
    const int nij = g.ni * g.nj, nt = blockDim.x;
    uint2* L = reinterpret_cast<uint2*>(sm);                 // planes * nij, by pass
    float* E = sm + 2 * (size_t)planes * nij;                // (planes + 2) * nij
    // per pass, for the sides towards lower and higher planes: unknowns in the neighbour's and in this CTA's
    // boundary plane
    __shared__ int cnt[8], start[9], halo[2][8], edge[2][8];
    __shared__ float dia_tab[64], unread;
    __shared__ __align__(8) unsigned long long bar[2];
    const Slab s = make_slab(g, planes, E);
    const int tid = threadIdx.x, own = s.np * nij, n0 = s.k0 * nij;
    const float c3[3] = {g.inv_dx[0] * g.inv_dx[0], g.inv_dx[1] * g.inv_dx[1], g.inv_dx[2] * g.inv_dx[2]};
    for (int x = tid; x < (s.np + 2) * nij; x += nt) E[x] = 0.f;
    if (tid < 64) dia_tab[tid] = mask_diag(c3, (unsigned)tid);
    if (tid < 8) cnt[tid] = halo[0][tid] = halo[1][tid] = edge[0][tid] = edge[1][tid] = 0;
    if (tid < 2) bar_init(&bar[tid]);
    const bool sx = g.periodic[0] && ((g.ni - 1) & 1), sy = g.periodic[1] && ((g.nj - 1) & 1),
               sz = g.periodic[2] && ((g.nk - 1) & 1);
    const int npass = 2 + 2 * ((int)sx + (int)sy + (int)sz);
    __syncthreads();
    // pass of a node: 0, 1 its colour, 2 m + colour on m seams (-1: no unknown); wraps: its wrap flags
    auto info = [&](int n, unsigned kd, unsigned& wraps) -> int {
        if ((kd & 3) != kFree) return -1;
        int i, j, k;
        node_ijk(g, n, i, j, k);
        const int m = (int)(sx && i == g.ni - 2) + (int)(sy && j == g.nj - 2) + (int)(sz && k == g.nk - 2);
        wraps = wrap_flags(g, i, j);
        return 2 * m + ((i + j + k) & 1);
    };
    unsigned wf;
    for (int x = tid; x < own; x += nt) {
        const int p = info(n0 + x, kind[n0 + x], wf);
        if (p < 0) continue;
        atomicAdd(&cnt[p], 1);
        if (x < nij) atomicAdd(&edge[0][p], 1);
        if (x >= own - nij) atomicAdd(&edge[1][p], 1);
    }
    for (int x = tid; x < 2 * nij; x += nt) {  // what the neighbours send in each pass
        const int n = halo_node(s, x);
        const int p = n >= 0 ? info(n, kind[n], wf) : -1;
        if (p >= 0) atomicAdd(&halo[x >= nij][p], 1);
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
    // the boundary planes first: their values are on their way while the inner planes are updated
    for (int inner = 0; inner < 2; inner++) {
        for (int x = tid; x < own; x += nt) {
            if ((x >= nij && x < own - nij) != (inner == 1)) continue;
            const unsigned kd = kind[n0 + x];
            const int p = info(n0 + x, kd, wf);
            if (p >= 0)
                L[atomicAdd(&cnt[p], 1)] =
                    make_uint2((unsigned)(x + nij) | ((kd >> 2) & 63u) << 20 | wf << 26, __float_as_uint(r[n0 + x]));
        }
        __syncthreads();
    }
    cluster_sync();  // every CTA's halo planes are zero, its barriers and lists are there
    unsigned phase = 0;  // bit b: parity of barrier b's next phase
    int q = 0;
    bool ok = true;
    for (int it = 0; it < sweeps && ok; it++)
        for (int p = 0; p < npass; p++, q ^= 1) {
            const unsigned lo_bar = s.has_lo ? map_rank(&bar[q], s.lo_rank) : 0u,
                           hi_bar = s.has_hi ? map_rank(&bar[q], s.hi_rank) : 0u;
            if (tid == 0) {
                const int words = (s.has_lo ? max(1, halo[0][p]) : 0) + (s.has_hi ? max(1, halo[1][p]) : 0);
                bar_expect(&bar[q], 4u * (unsigned)words);
                if (s.has_lo && !edge[0][p]) st_async(map_rank(&unread, s.lo_rank), 0.f, lo_bar);
                if (s.has_hi && !edge[1][p]) st_async(map_rank(&unread, s.hi_rank), 0.f, hi_bar);
            }
            const float om = p < 2 ? omega : 1.0f;
            for (int y = start[p] + tid; y < start[p + 1]; y += nt) {
                const uint2 u = L[y];
                const int idx = (int)(u.x & 0xFFFFFu);
                int o[6];
                plane_nb(g, u.x >> 26, o[0], o[1], o[2], o[3]);
                o[4] = -nij;
                o[5] = nij;
                float off = 0.f;
#pragma unroll
                for (int d = 0; d < 6; d++) off += c3[d >> 1] * E[idx + o[d]];
                const float en = E[idx];
                put(s, E, idx, en + om * ((__uint_as_float(u.y) + off) / dia_tab[(u.x >> 20) & 63u] - en), lo_bar, hi_bar);
            }
            const bool got = bar_wait(&bar[q], phase >> q & 1u, wait.polls);
            phase ^= 1u << q;
            if (__syncthreads_or(!got)) {
                ok = false;
                break;
            }
        }
    if (!ok && tid == 0) {
        set_error(wait.err, kErrBarrierTimeout);
        *wait.fail = 1;
    }
    for (int x = tid; x < own; x += nt) e[n0 + x] = E[nij + x];
    if (s.k0 + s.np == s.nz)  // the copy plane of a periodic z axis holds no unknown
        for (int x = s.nz * nij + tid; x < g.nv; x += nt) e[x] = 0.f;
    cluster_leave(!ok);
}

// ------------------------------------------------------------------------------------
// the whole inner CG solve of L e = r from e = 0 (the iteration of k_pcg_k1 / k_pcg_k2)
// ------------------------------------------------------------------------------------
// Sums of N per-thread values over the cluster, times scale, in every lane of warp 0 of every CTA, float-float
// (48 bits) in a fixed order (scale and what rounds as in grid_total).  Every warp sends its
// partials straight to all CTAs (red, counted on bar), so a sum is one message deep and costs no block
// barrier.  FP64 is kept out of this chain: its adds and above all its divides run on a pipe so narrow
// here that they were a third of an iteration.  False when the partials did not arrive in time.
template <int N, int NW>
__device__ __forceinline__ bool cluster_sum(const FF (&v)[N], const float (&scale)[N], float2 (*red)[kMaxCtas * NW], int ctas,
                                            unsigned long long* bar, unsigned parity, long long polls, FF (&out)[N]) {
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
    if (threadIdx.x == 0) bar_expect(bar, 8u * N * NW * (unsigned)ctas);
    const FF x = warp_halved(v);
    FF p[N];
#pragma unroll
    for (int c = 0; c < N; c++)
        p[c] = FF{__shfl_sync(0xffffffffu, x.hi, warp_home<N>(c)) * scale[c], __shfl_sync(0xffffffffu, x.lo, warp_home<N>(c)) * scale[c]};
    if (lane < ctas) {
        const unsigned rb = map_rank(bar, (unsigned)lane);
#pragma unroll
        for (int c = 0; c < N; c++)
            st_async2(map_rank(&red[c][cluster_rank() * NW + wp], (unsigned)lane), p[c].hi, p[c].lo, rb);
    }
    if (wp != 0) return true;
    const bool ok = bar_wait(bar, parity, polls);
    __syncwarp();
#pragma unroll
    for (int c = 0; c < N; c++) out[c] = FF{0.f, 0.f};
    for (int y = lane; y < ctas * NW; y += 32)
#pragma unroll
        for (int c = 0; c < N; c++) out[c] = ff_gather(out[c], FF{red[c][y].x, red[c][y].y});
    warp_total(out);
    return ok;
}

// flag[0]: converged (r.r <= target), flag[1]: iterations done.  A thread keeps K nodes (x = tid + m NT of
// the CTA's planes) in registers: r, e, q, mask; only d is shared.  The three barriers count the halo planes
// of d, the partials of d.q and those of the three sums after the update; each completes once per
// iteration, and a CTA can only be one of them ahead of another, so no slot is written before its last
// value was read.
template <int NT, int K>
__global__ void __launch_bounds__(NT, 1) k_pcg_cluster(GridDev g, float* __restrict__ e, const float* __restrict__ r,
                                                       const uint16_t* __restrict__ kind, SumScales sc, FF target, int cap,
                                                       int planes, int* flag, ClusterWait wait) {
    constexpr int NW = NT / 32;
    const float sc1[1] = {sc.rz}, sc3[3] = {sc.rz, sc.rz, sc.rr};
    extern __shared__ __align__(16) float sm[];
    float* D = sm;  // direction, (planes + 2) * nij
    __shared__ float2 red1[1][kMaxCtas * NW], red3[3][kMaxCtas * NW];
    __shared__ __align__(8) unsigned long long bar_d, bar_1, bar_3;
    __shared__ float inv_tab[64], dia_tab[64];
    __shared__ float s_alpha, s_beta;
    __shared__ int s_stop, s_halo;  // s_stop: 1 finished, 2 a wait ran out
    const int nij = g.ni * g.nj;
    const Slab s = make_slab(g, planes, D);
    const int tid = threadIdx.x, own = s.np * nij, n0 = s.k0 * nij;
    const int ctas = (s.nz + planes - 1) / planes;
    const float c3[3] = {g.inv_dx[0] * g.inv_dx[0], g.inv_dx[1] * g.inv_dx[1], g.inv_dx[2] * g.inv_dx[2]};
    if (tid < 64) {
        dia_tab[tid] = mask_diag(c3, (unsigned)tid);
        inv_tab[tid] = 1.f / dia_tab[tid];
    }
    if (tid == 0) {
        bar_init(&bar_d);
        bar_init(&bar_1);
        bar_init(&bar_3);
        s_beta = 0.f;
        s_stop = s_halo = 0;
    }
    for (int x = tid; x < (s.np + 2) * nij; x += NT) D[x] = 0.f;
    __syncthreads();
    static_assert(K <= kFp32Nodes, "a thread's FP32 sums");
    float R[K], X[K], Q[K], f = 0.f;
    unsigned M[K];  // 0: no unknown; bit 0 set, mirror mask (6 bits), wrap flags (4 bits)
#pragma unroll
    for (int m = 0; m < K; m++) {
        const int x = tid + m * NT;
        R[m] = X[m] = Q[m] = 0.f;
        M[m] = 0u;
        if (x >= own) continue;
        const unsigned kd = kind[n0 + x];
        if ((kd & 3) != kFree) continue;
        int i, j, k;
        node_ijk(g, n0 + x, i, j, k);
        M[m] = 1u | ((kd >> 2) & 63u) << 1 | wrap_flags(g, i, j) << 7;
        R[m] = r[n0 + x];
        f += R[m] * (R[m] * inv_tab[(kd >> 2) & 63u]);
    }
    for (int x = tid; x < 2 * nij; x += NT) {
        const int n = halo_node(s, x);
        if (n >= 0 && (kind[n] & 3) == kFree) atomicAdd(&s_halo, 1);
    }
    cluster_sync();  // every CTA's halo planes are zero and its barriers are there
    FF t1[1], t3[3], rz;
    unsigned ph3 = 0, ph = 0;
    const FF v0[3] = {FF{f, 0.f}, FF{0.f, 0.f}, FF{0.f, 0.f}};
    bool ok = cluster_sum<3, NW>(v0, sc3, red3, ctas, &bar_3, ph3, wait.polls, t3);  // r.z
    ph3 ^= 1u;
    rz = t3[0];
    if (tid == 0 && !ok) s_stop = 2;
    __syncthreads();
    const unsigned lo_bar = s.has_lo ? map_rank(&bar_d, s.lo_rank) : 0u, hi_bar = s.has_hi ? map_rank(&bar_d, s.hi_rank) : 0u;
    int it = 0;
    while (it < cap && !s_stop) {
        // d = z + beta d
        if (tid == 0) bar_expect(&bar_d, 4u * (unsigned)s_halo);
        const float beta = s_beta;
#pragma unroll
        for (int m = 0; m < K; m++) {
            if (!M[m]) continue;
            const int x = tid + m * NT + nij;
            put(s, D, x, R[m] * inv_tab[(M[m] >> 1) & 63u] + beta * D[x], lo_bar, hi_bar);
        }
        const bool got = bar_wait(&bar_d, ph, wait.polls);
        if (__syncthreads_or(!got)) {
            s_stop = 2;
            break;
        }
        // q = L d, d.q
        float f1 = 0.f;
#pragma unroll
        for (int m = 0; m < K; m++) {
            if (!M[m]) continue;
            int o[6];
            plane_nb(g, M[m] >> 7, o[0], o[1], o[2], o[3]);
            o[4] = -nij;
            o[5] = nij;
            const float* dp = D + nij + tid + m * NT;
            float off = 0.f;
#pragma unroll
            for (int d = 0; d < 6; d++) off += c3[d >> 1] * dp[o[d]];  // zero on MIRROR and FIXED nodes
            const float dn = dp[0];
            Q[m] = dia_tab[(M[m] >> 1) & 63u] * dn - off;
            f1 += dn * Q[m];
        }
        const FF v1[1] = {FF{f1, 0.f}};
        ok = cluster_sum<1, NW>(v1, sc1, red1, ctas, &bar_1, ph, wait.polls, t1);
        if (tid == 0) {
            s_alpha = t1[0].hi != 0.f ? ff_ratio(rz, t1[0]) : 0.f;
            if (!ok) s_stop = 2;
        }
        __syncthreads();
        if (s_stop) break;
        // e += alpha d, r -= alpha q, z = r / D
        const float alpha = s_alpha;
        float f3[3] = {0.f, 0.f, 0.f};
#pragma unroll
        for (int m = 0; m < K; m++) {
            if (!M[m]) continue;
            const float inv = inv_tab[(M[m] >> 1) & 63u];
            X[m] += alpha * D[tid + m * NT + nij];
            const float ro = R[m];
            const float rn = ro - alpha * Q[m];
            const float zn = rn * inv;
            f3[0] += rn * zn;
            f3[1] += rn * (ro * inv);
            f3[2] += rn * rn;
            R[m] = rn;
        }
        const FF v3[3] = {FF{f3[0], 0.f}, FF{f3[1], 0.f}, FF{f3[2], 0.f}};
        ok = cluster_sum<3, NW>(v3, sc3, red3, ctas, &bar_3, ph3, wait.polls, t3);
        it++;
        if (tid == 0) {
            const float over = (t3[2].hi - target.hi) + (t3[2].lo - target.lo);
            if (!ok) s_stop = 2;
            else if (!(over > 0.f)) s_stop = over <= 0.f ? 1 : 3;  // converged, or not a number
            s_beta = ff_ratio(ff_add(t3[0], ff_neg(t3[1])), rz);
        }
        rz = t3[0];
        ph ^= 1u;
        ph3 ^= 1u;
        __syncthreads();
    }
    __syncthreads();
    if (tid == 0) {
        if (s.k0 == 0) {
            flag[0] = s_stop == 1;
            flag[1] = it;
        }
        if (s_stop == 2) {
            set_error(wait.err, kErrBarrierTimeout);
            *wait.fail = 1;
        }
    }
#pragma unroll
    for (int m = 0; m < K; m++)
        if (tid + m * NT < own) e[n0 + tid + m * NT] = X[m];
    if (s.k0 + s.np == s.nz)
        for (int x = s.nz * nij + tid; x < g.nv; x += NT) e[x] = 0.f;
    cluster_leave(s_stop == 2);
}

size_t sor_smem(long nij, int planes) { return 4 * nij * (3 * (long)planes + 2); }
size_t pcg_smem(long nij, int planes) { return 4 * nij * ((long)planes + 2); }

void fill_config(int ctas, int threads, size_t smem, cudaStream_t s, cudaLaunchConfig_t& cfg,
                 cudaLaunchAttribute* at) {
    cfg = cudaLaunchConfig_t{};
    cfg.gridDim = dim3((unsigned)ctas);
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)ctas;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
}
constexpr size_t kSmemMost = 216 * 1024;  // with the static arrays below the 227 KB of a CTA
// nodes per CTA up to which one cluster is the faster form: at 45^3 (6075 a CTA) 25 sweeps take 101 us here
// and 108 us on the whole GPU (pic_persist.cu), a CG iteration 6.0 and 7.4 us; at 31 x 31 x 51 (3844) 71
// and 104 us, 4.6 and 7.3 us; sweeps of 60^3 (14 400) 161 and 116 us
constexpr long kOwnMost = 6144;
int stack_planes(const GridDev& g) { return g.periodic[2] ? g.nk - 1 : g.nk; }
// whether a cluster of the kernel can be resident (its attributes are set here, before any launch)
template <class K>
bool fits(K kernel, int ctas, int threads, size_t smem) {
    cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemMost);
    cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute at[1];
    fill_config(ctas, threads, smem, 0, cfg, at);
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) == cudaSuccess && n > 0) return true;
    cudaGetLastError();  // a cluster of this size does not fit this GPU
    return false;
}
using PcgKernel = void (*)(GridDev, float*, const float*, const uint16_t*, SumScales, FF, int, int, int*, ClusterWait);
// the smallest form whose registers hold a CTA's nodes
PcgKernel pcg_kernel(long own, int* threads) {
    *threads = own <= 2048 ? 256 : 512;
    if (own <= 512) return k_pcg_cluster<256, 2>;
    if (own <= 1024) return k_pcg_cluster<256, 4>;
    if (own <= 2048) return k_pcg_cluster<256, 8>;
    if (own <= 4096) return k_pcg_cluster<512, 8>;
    if (own <= 6144) return k_pcg_cluster<512, 12>;
    return nullptr;
}
// threads of the sweeps: one listed node of a pass each, where that many fit
int sor_threads(long own) { return (int)std::min<long>(1024, std::max<long>(128, (own / 2 + 31) / 32 * 32)); }
}  // namespace

int plan_sor_cluster(const GridDev& g, int most) {
    const int nz = stack_planes(g);
    const long nij = (long)g.ni * g.nj;
    for (int c = most; c >= 1; c >>= 1) {
        const int planes = (nz + c - 1) / c, ctas = (nz + planes - 1) / planes;
        const size_t b = sor_smem(nij, planes);
        if (b > kSmemMost || nij * planes > kOwnMost) return 0;
        if (fits(k_sor_cluster, ctas, sor_threads(nij * planes), b)) return planes;
    }
    return 0;
}
int plan_pcg_cluster(const GridDev& g, int most) {
    const int nz = stack_planes(g);
    const long nij = (long)g.ni * g.nj;
    for (int c = most; c >= 1; c >>= 1) {
        const int planes = (nz + c - 1) / c, ctas = (nz + planes - 1) / planes;
        const size_t b = pcg_smem(nij, planes);
        int threads;
        PcgKernel k = pcg_kernel(nij * planes, &threads);
        if (!k || b > kSmemMost || nij * planes > kOwnMost) return 0;
        if (fits(k, ctas, threads, b)) return planes;
    }
    return 0;
}

void launch_sor_cluster(const GridDev& g, SolveWork& w, float omega, int sweeps, int planes, cudaStream_t s) {
    const long nij = (long)g.ni * g.nj;
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute at[1];
    fill_config((stack_planes(g) + planes - 1) / planes, sor_threads(nij * planes), sor_smem(nij, planes), s, cfg, at);
    cudaLaunchKernelEx(&cfg, k_sor_cluster, g, w.e, (const float*)w.r, reinterpret_cast<const uint16_t*>(w.kind), omega,
                       sweeps, planes, ClusterWait{w.wait_polls, w.err, w.flag + 2});
}
void launch_pcg_cluster(const GridDev& g, SolveWork& w, double r2, double target_rr, int cap, int planes, cudaStream_t s) {
    const long nij = (long)g.ni * g.nj;
    int threads;
    PcgKernel k = pcg_kernel(nij * planes, &threads);
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute at[1];
    fill_config((stack_planes(g) + planes - 1) / planes, threads, pcg_smem(nij, planes), s, cfg, at);
    const SumScales sc = sum_scales(g, r2);
    cudaLaunchKernelEx(&cfg, k, g, w.e, (const float*)w.r, reinterpret_cast<const uint16_t*>(w.kind), sc,
                       ff_from_double(target_rr * sc.rr), cap, planes, w.flag, ClusterWait{w.wait_polls, w.err, w.flag + 2});
}

}  // namespace pic
