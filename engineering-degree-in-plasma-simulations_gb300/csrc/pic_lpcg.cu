// The whole inner solve of the learned-preconditioned flexible CG as one persistent kernel, for grids whose
// solver arrays stay in L2.
//
// One iteration as launches (k_lpcg_k1, k_lpcg_k2, the level kernels, k_lp_up0_pipe) is about ten kernels of
// 6 to 28 us on a grid of a million nodes, none of which is bound by anything but latency: launch and drain,
// the first fetch of each kernel's instructions, and one pass of dependent reads.  Here one cooperative
// launch runs the iterations until the residual meets the target; the instructions stay cached, and phases
// are separated by grid barriers.  Fine-grid phases work on tiles of 32 x 8 x 8 nodes that a CTA owns for
// the whole solve: the tile and its halo are read into registers while the tile before is computed from
// shared memory.  An iteration is
//   coarse levels   z_2 .. , e_2 from z_1 (lp_coarse_levels)
//   level 1         e_1 = op(z_1) + P e_2
//   fine level      z = mask (S0 r + P e_1), z.r, z.q
//   direction       d = z + beta d, q = L d, d.q                  (beta = -z.q / d.q of the iteration before)
//   update          r -= alpha q, e += alpha d, r.r, and z_1 = R r of the new residual in the same pass
// Directions and residuals alternate between two buffers, since a tile's halo is still being read by its
// neighbours when it is updated.  The arithmetic of a node is that of the kernels above.
//
// What bounds it: the latency of a tile's dependent reads and shared-memory passes (16 warps an SM, issue
// slots 27 % busy), five barriers of 1.3 us, and the coarse levels (20 of 68 us).  1024 threads a CTA spill at
// 64 registers: 85 us.  One iteration of 64 x 64 x 256 nodes: 95 us as launches, 68 us here; a loop of 20
// steps on it 33.2 -> 26.8 ms.
#include <algorithm>
#include "pic_lp_levels.cuh"

namespace pic {
namespace {

constexpr int kThr = kLvThr;
constexpr int kTX = 32, kTY = 8, kTZ = 8, kTile = kTX * kTY * kTZ;  // a thread: four nodes of a z column
constexpr int kHY = kTY + 2, kHZ = kTZ + 2, kRows = kHY * kHZ;
constexpr int kP = 36;                                     // pitch of a staged row
constexpr int kWarps = kThr / 32, kRowsPer = (kRows + kWarps - 1) / kWarps;
constexpr int kCX = kTX / 2 + 2, kCY = kTY / 2 + 2, kCZ = kTZ / 2 + 2, kCTile = kCX * kCY * kCZ;
constexpr int kMostRounds = 16;                            // tiles a CTA owns
// The tiles of a CTA are serial, while the launches fill the SMs better the more tiles there are: a loop of
// 1.0 M nodes spends 15.6 ms in solves here and 18.7 as launches, one of 2.1 M nodes 12.6 and 11.5; the line lies between.
constexpr int kLpcgMostNodes = 3 << 19;
struct LpcgArgs {
    GridDev g;
    LpCoarseLevels lev;    // from level 2 on; from 1 on where level 1 is the dense one
    LView f, z1, e1, e2;   // level 0 (no array), level 1; e2.a null: one level only
    float *r[2], *d[2], *z, *q, *e;
    const uint16_t* kind;
    const float* S0;
    SumScales sc;
    FF target;
    int cap, tx_n, ty_n, ntiles, rounds;
    int* flag;
    GridSync* sync;
    GridWait wait;
};

// a tile's origin
struct TileAt {
    int x0, y0, z0;
};
__device__ __forceinline__ TileAt tile_at(const LpcgArgs& a, int tile) {
    const int bx = tile % a.tx_n, t = tile / a.tx_n;
    return TileAt{bx * kTX, (t % a.ty_n) * kTY, (t / a.ty_n) * kTZ};
}
// one value per staged point of a tile and its halo, read into registers: rows wp, wp + kWarps, ... of the
// kHY x kHZ rows, a lane the row's point `lane` (lanes 0 and 1 also points 32, 33).  tab: the offsets of the
// tile's rows (-1: outside, zero), ox, ox2: those of the lane's points; ld: the value at a node offset
struct Staged {
    float v[kRowsPer], v2[kRowsPer];
};
template <class LD>
__device__ __forceinline__ void stage_read(const int* tab, int ox, int ox2, Staged& s, LD ld) {
    const int wp = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < kRowsPer; k++) {
        const int row = wp + k * kWarps;
        const int o = row < kRows ? tab[row] : -1;
        s.v[k] = (o | ox) >= 0 ? ld(o + ox) : 0.f;
        s.v2[k] = (o | ox2) >= 0 ? ld(o + ox2) : 0.f;
    }
}
__device__ __forceinline__ void stage_write(float* T, const Staged& s) {
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < kRowsPer; k++) {
        const int row = wp + k * kWarps;
        if (row >= kRows) continue;
        T[row * kP + lane] = s.v[k];
        if (lane < 2) T[row * kP + 32 + lane] = s.v2[k];
    }
}

// flag[0]: converged (r.r <= target), flag[1]: iterations done.  LONG: some CTA owns more than kRun tiles, so that
// a thread's FP32 sums are cut into runs
constexpr int kRun = kFp32Nodes / 4;  // tiles
template <bool LONG>
__global__ void __launch_bounds__(kThr, 1) k_lpcg_grid(const __grid_constant__ LpcgArgs a) {
    extern __shared__ __align__(16) float dyn[];
    LevelSmem& sm = *reinterpret_cast<LevelSmem*>(dyn);
    float* T = dyn + sizeof(LevelSmem) / 4;              // two staged tiles
    float* E1 = sm.tile;                                 // the fine level's tile of e_1
    int* tabS = reinterpret_cast<int*>(T + 2 * kRows * kP);  // row offsets of the CTA's tiles: stencil rule,
    int* tabR = tabS + a.rounds * kRows;                     // restriction rule
    int4* org = reinterpret_cast<int4*>(tabR + a.rounds * kRows);  // origins of the CTA's tiles
    unsigned char* F = reinterpret_cast<unsigned char*>(org + a.rounds);  // node flags: FREE 128, mirrors
    __shared__ float S[27], dia[64], s_alpha, s_beta;
    __shared__ float2 wsum[2][kThr / 32], runs[2][LONG ? kThr : 1];
    __shared__ int s_fail, s_stop;
    static_assert(kCTile <= kLvTile, "the tile of e_1 shares the level tile's place");
    const GridDev& g = a.g;
    const float sc_rr[1] = {a.sc.rr}, sc_dq[1] = {a.sc.rz}, sc_z[2] = {a.sc.rz, a.sc.rz};
    const int tid = threadIdx.x, tx = tid & 31, ty = (tid >> 5) & 7, tz = (tid >> 8) * 4;
    const float c3[3] = {g.inv_dx[0] * g.inv_dx[0], g.inv_dx[1] * g.inv_dx[1], g.inv_dx[2] * g.inv_dx[2]};
    if (tid < 27) S[tid] = a.S0[tid];
    if (tid < 64) {
        float dg = 0.f;
        for (int d = 0; d < 6; d++)
            if (!(tid & (1 << d))) dg += c3[d >> 1];
        dia[tid] = dg;
    }
    if (tid == 0) {
        s_fail = s_stop = 0;
        s_alpha = s_beta = 0.f;
    }
    if (tid == 0) sm.lev = a.lev;  // once a solve: lp_load_levels measured 1 % slower here
    for (int l = 1; l < a.lev.ld && l <= kLpNetLevels; l++)
        for (int x = tid; x < 27 * 128; x += kThr) {
            const int cls = x >> 7, dd = x & 127;
            sm.k5[l - 1][cls][dd] = dd < 125 ? a.lev.fold[l][kLpFold + 125 * cls + dd] : 0.f;
        }
    // zero what is only written on unknowns, and the flags of the CTA's tiles
    for (int n = blockIdx.x * kThr + tid; n < g.nv; n += gridDim.x * kThr) a.e[n] = a.z[n] = a.q[n] = a.d[0][n] = a.d[1][n] = 0.f;
    auto node = [&](const TileAt& t, int k) { return ((t.z0 + tz + k) * g.nj + t.y0 + ty) * g.ni + t.x0 + tx; };
    auto inside = [&](const TileAt& t, int k) {
        return t.x0 + tx < a.f.n[0] && t.y0 + ty < a.f.n[1] && t.z0 + tz + k < a.f.n[2];
    };
    for (int q = 0; q < a.rounds; q++) {
        const int tile = blockIdx.x + q * gridDim.x;
        const TileAt t = tile_at(a, min(tile, a.ntiles - 1));
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const unsigned kd = tile < a.ntiles && inside(t, k) ? a.kind[node(t, k)] : (unsigned)kFixed;
            F[(q * 4 + k) * kThr + tid] = (kd & 3) == kFree ? (unsigned char)(128u | ((kd >> 2) & 63u)) : (unsigned char)0;
        }
    }
    for (int i = tid; i < a.rounds * kRows; i += kThr) {
        const int q = i / kRows, row = i - q * kRows;
        const TileAt t = tile_at(a, min((int)(blockIdx.x + q * gridDim.x), a.ntiles - 1));
        const int uy = t.y0 - 1 + row % kHY, uz = t.z0 - 1 + row / kHY;
        const int sy = lv_map(uy, a.f.n[1], a.f.per[1]), sz = lv_map(uz, a.f.n[2], a.f.per[2]);
        const int ry = rs_map(uy, a.f, a.z1, 1), rz = rs_map(uz, a.f, a.z1, 2);
        tabS[i] = (sy | sz) < 0 ? -1 : sy * a.f.sy + sz * a.f.sz;
        tabR[i] = (ry | rz) < 0 ? -1 : ry * a.f.sy + rz * a.f.sz;
    }
    if (tid < a.rounds) {
        const TileAt t = tile_at(a, min((int)(blockIdx.x + tid * gridDim.x), a.ntiles - 1));
        org[tid] = make_int4(t.x0, t.y0, t.z0, 0);
    }
    auto at = [&](int round) {
        const int4 o = org[round];
        return TileAt{o.x, o.y, o.z};
    };
    const int mine = ((int)a.ntiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;  // tiles of this CTA
    const int lane = tid & 31;
    auto sx = [&](int u) { return lv_map(u, a.f.n[0], a.f.per[0]); };
    auto rx = [&](int u) { return rs_map(u, a.f, a.z1, 0); };
    __syncthreads();
    unsigned target = 0;
    FF dq[1] = {FF{0.f, 0.f}}, rr[1], zz[2], rz{0.f, 0.f};
    int it = 0, rc = 0, dc = 0;  // r[rc], d[dc]: the residual and the last direction

    // The FP32 sum f of a thread's columns of four nodes joins its pair runs[c] every kFp32Nodes nodes; whole_run is the
    // pair at the end.  In shared memory: pairs in registers cost 3 us an iteration of a million nodes in spills.
    auto run = [&](int round, int c, float& f) {
        if (!LONG || (round + 1) % kRun || round + 1 >= mine) return;
        const float2 p = round + 1 == kRun ? make_float2(0.f, 0.f) : runs[c][tid];
        const FF s = ff_acc(FF{p.x, p.y}, f);
        runs[c][tid] = make_float2(s.hi, s.lo);
        f = 0.f;
    };
    auto whole_run = [&](int c, float f) {
        const float2 p = LONG && mine > kRun ? runs[c][tid] : make_float2(0.f, 0.f);
        return ff_acc(FF{p.x, p.y}, f);
    };
    // r -= alpha q (into r[rc ^ 1]), e += alpha d, r.r, z_1 = R r; the first time only z_1 of r[0]
    auto update = [&](bool first) {
        const float alpha = s_alpha;
        const float* r = a.r[rc];
        const float* d = a.d[dc];
        float* rn = a.r[rc ^ 1];
        float f = 0.f;
        Staged s;
        float ev[4], dv[4];
        auto read = [&](int round) {
            const TileAt t = at(round);
            const int ox = rx(t.x0 - 1 + lane), ox2 = lane < 2 ? rx(t.x0 + 31 + lane) : -1;
            if (first)
                stage_read(tabR + round * kRows, ox, ox2, s, [&](int o) { return __ldcg(r + o); });
            else
                stage_read(tabR + round * kRows, ox, ox2, s,
                           [&](int o) { return __ldcg(r + o) - alpha * __ldcg(a.q + o); });
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const bool in = !first && inside(t, k);
                ev[k] = in ? __ldcg(a.e + node(t, k)) : 0.f;
                dv[k] = in ? __ldcg(d + node(t, k)) : 0.f;
            }
        };
        if (mine > 0) read(0);
        for (int round = 0; round < mine; round++) {
            float* Tb = T + (round & 1) * kRows * kP;
            const TileAt t = at(round);
            stage_write(Tb, s);
            float en[4];
#pragma unroll
            for (int k = 0; k < 4; k++) en[k] = ev[k] + alpha * dv[k];
            __syncthreads();
            if (round + 1 < mine) read(round + 1);
            if (!first) {
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    if (!inside(t, k)) continue;
                    const float v = Tb[((tz + k + 1) * kHY + ty + 1) * kP + tx + 1];
                    f += v * v;
                    rn[node(t, k)] = v;
                    a.e[node(t, k)] = en[k];
                }
                run(round, 0, f);
            }
            // 16 x 4 x 4 coarse voxels, two threads each (two of the four fine planes)
            const int v = tid >> 1, i = v & 15, j = (v >> 4) & 3, k = v >> 6, h = tid & 1;
            const float* p = Tb + ((2 * k + 2 * h) * kHY + 2 * j) * kP + 2 * i;
            float sum = 0.f;
#pragma unroll
            for (int kz = 0; kz < 2; kz++) {
                float az = 0.f;
#pragma unroll
                for (int ky = 0; ky < 4; ky++) {
                    const float* row = p + (kz * kHY + ky) * kP;
                    az += ((ky == 0 || ky == 3) ? 0.25f : 0.75f) *
                          (0.25f * row[0] + 0.75f * row[1] + 0.75f * row[2] + 0.25f * row[3]);
                }
                sum += (h == kz ? 0.25f : 0.75f) * az;
            }
            sum += __shfl_xor_sync(0xffffffffu, sum, 1);
            const int cx = (t.x0 >> 1) + i, cy = (t.y0 >> 1) + j, cz = (t.z0 >> 1) + k;
            if (h == 0 && cx < a.z1.n[0] && cy < a.z1.n[1] && cz < a.z1.n[2]) a.z1.a[lv_off(a.z1, cx, cy, cz)] = sum;
        }
        const FF acc[1] = {whole_run(0, f)};
        return grid_total<1, kThr>(acc, sc_rr, wsum, a.sync->part + 1, a.wait, target, &s_fail, rr);
    };

    bool ok = grid_barrier(a.wait, target, &s_fail);  // the zeros are there
    ok = ok && update(true);
    while (ok && it < a.cap) {
        // ---- z = B r
        if (a.lev.ld == 1) {
            lp_dense_level(sm.lev, sm.tile);
        } else {
            if (a.lev.m < a.lev.nlev)
                ok = lp_coarse_levels<false>(sm.lev, sm, a.wait, target, &s_fail) && grid_barrier(a.wait, target, &s_fail);
            if (!ok) break;
            lp_net_level<false, false>(a.z1, a.e2, a.e1, sm.k5[0], sm, blockIdx.x, gridDim.x);
        }
        if (!(ok = grid_barrier(a.wait, target, &s_fail))) break;
        {
            const float* r = a.r[rc];
            float w[27], f[2] = {0.f, 0.f};
#pragma unroll
            for (int m = 0; m < 27; m++) w[m] = S[m];
            Staged s;
            float qv[4], ev[(kCTile + kThr - 1) / kThr];
            auto read = [&](int round) {
                const TileAt t = at(round);
                stage_read(tabS + round * kRows, sx(t.x0 - 1 + lane), lane < 2 ? sx(t.x0 + 31 + lane) : -1, s,
                           [&](int o) { return __ldcg(r + o); });
#pragma unroll
                for (int k = 0; k < (kCTile + kThr - 1) / kThr; k++) {
                    const int i = tid + k * kThr;
                    const int ux = lv_map(t.x0 / 2 - 1 + i % kCX, a.e1.n[0], a.e1.per[0]);
                    const int uy = lv_map(t.y0 / 2 - 1 + i / kCX % kCY, a.e1.n[1], a.e1.per[1]);
                    const int uz = lv_map(t.z0 / 2 - 1 + i / (kCX * kCY), a.e1.n[2], a.e1.per[2]);
                    ev[k] = i < kCTile && ux >= 0 && uy >= 0 && uz >= 0 ? __ldcg(a.e1.a + lv_off(a.e1, ux, uy, uz)) : 0.f;
                }
#pragma unroll
                for (int k = 0; k < 4; k++) qv[k] = inside(t, k) ? __ldcg(a.q + node(t, k)) : 0.f;
            };
            if (mine > 0) read(0);
            for (int round = 0; round < mine; round++) {
                float* Tb = T + (round & 1) * kRows * kP;
                const TileAt t = at(round);
                stage_write(Tb, s);
                if (round) __syncthreads();  // the tile of e_1 before has been read
#pragma unroll
                for (int k = 0; k < (kCTile + kThr - 1) / kThr; k++)
                    if (tid + k * kThr < kCTile) E1[tid + k * kThr] = ev[k];
                const float q0[4] = {qv[0], qv[1], qv[2], qv[3]};
                __syncthreads();
                if (round + 1 < mine) read(round + 1);
                // x-y interpolation of the column's four coarse planes (tile origins are even)
                float px[4];
                {
                    const int lx = (tx >> 1) + 1, ly = (ty >> 1) + 1, gx = (tx & 1) ? 1 : -1, gy = (ty & 1) ? 1 : -1;
#pragma unroll
                    for (int c = 0; c < 4; c++) {
                        const float* C = E1 + ((tz >> 1) + c) * kCX * kCY;
                        const float a0 = 0.75f * C[ly * kCX + lx] + 0.25f * C[ly * kCX + lx + gx];
                        const float a1 = 0.75f * C[(ly + gy) * kCX + lx] + 0.25f * C[(ly + gy) * kCX + lx + gx];
                        px[c] = 0.75f * a0 + 0.25f * a1;
                    }
                }
                float Pr = 0.f, Qr = 0.f;
#pragma unroll
                for (int hz = 0; hz < 6; hz++) {
                    float a0 = 0.f, a1 = 0.f, a2 = 0.f;
#pragma unroll
                    for (int dy = 0; dy < 3; dy++)
#pragma unroll
                        for (int dx = 0; dx < 3; dx++) {
                            const float v = Tb[((tz + hz) * kHY + ty + dy) * kP + tx + dx];
                            const int m = 3 * dy + dx;
                            a0 = fmaf(w[m], v, a0);
                            a1 = fmaf(w[9 + m], v, a1);
                            a2 = fmaf(w[18 + m], v, a2);
                        }
                    const int k = hz - 2;  // complete after plane k + 2
                    if (k >= 0 && (F[(round * 4 + k) * kThr + tid] & 128)) {
                        const int lz = 1 + (k >> 1), sz = (k & 1) ? 1 : -1;
                        const float v = Pr + a2 + (0.75f * px[lz] + 0.25f * px[lz + sz]);
                        a.z[node(t, k)] = v;
                        f[0] += v * Tb[((tz + k + 1) * kHY + ty + 1) * kP + tx + 1];
                        f[1] += v * q0[k];
                    }
                    Pr = Qr + a1;
                    Qr = a0;
                }
                run(round, 0, f[0]);
                run(round, 1, f[1]);
            }
            const FF acc[2] = {whole_run(0, f[0]), whole_run(1, f[1])};
            ok = grid_total<2, kThr>(acc, sc_z, wsum, a.sync->part + 2, a.wait, target, &s_fail, zz);  // z.r, z.q
        }
        if (tid == 0) s_beta = it > 0 && dq[0].hi != 0.f ? -ff_ratio(zz[1], dq[0]) : 0.f;
        rz = zz[0];
        __syncthreads();
        if (!ok) break;
        // ---- d = z + beta d (into d[dc ^ 1]), q = L d
        {
            const float beta = s_beta;
            const float* d = a.d[dc];
            float* dn = a.d[dc ^ 1];
            float f = 0.f;
            Staged s;
            auto read = [&](int round) {
                const int x0 = at(round).x0;
                stage_read(tabS + round * kRows, sx(x0 - 1 + lane), lane < 2 ? sx(x0 + 31 + lane) : -1, s,
                           [&](int o) { return __ldcg(a.z + o) + beta * __ldcg(d + o); });
            };
            if (mine > 0) read(0);
            for (int round = 0; round < mine; round++) {
                float* Tb = T + (round & 1) * kRows * kP;
                const TileAt t = at(round);
                stage_write(Tb, s);
                __syncthreads();
                if (round + 1 < mine) read(round + 1);
                const float* p = Tb + (tz * kHY + ty + 1) * kP + tx + 1;
                float c[6];
#pragma unroll
                for (int k = 0; k < 6; k++) c[k] = p[k * kHY * kP];
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    const unsigned fl = F[(round * 4 + k) * kThr + tid];
                    if (!fl) continue;
                    const float* pk = p + (k + 1) * kHY * kP;
                    float off = c3[0] * pk[-1];  // zero on MIRROR and FIXED nodes
                    off += c3[0] * pk[1];
                    off += c3[1] * pk[-kP];
                    off += c3[1] * pk[kP];
                    off += c3[2] * c[k];
                    off += c3[2] * c[k + 2];
                    const float qn = dia[fl & 63u] * c[k + 1] - off;
                    f += c[k + 1] * qn;
                    dn[node(t, k)] = c[k + 1];
                    a.q[node(t, k)] = qn;
                }
                run(round, 0, f);
            }
            const FF acc[1] = {whole_run(0, f)};
            ok = grid_total<1, kThr>(acc, sc_dq, wsum, a.sync->part, a.wait, target, &s_fail, dq);
        }
        if (tid == 0) s_alpha = dq[0].hi != 0.f ? ff_ratio(rz, dq[0]) : 0.f;
        __syncthreads();
        if (!ok) break;
        dc ^= 1;
        ok = update(false);
        rc ^= 1;
        it++;
        if (tid == 0) {
            const float over = (rr[0].hi - a.target.hi) + (rr[0].lo - a.target.lo);
            if (!(over > 0.f)) s_stop = over <= 0.f ? 1 : 3;
        }
        __syncthreads();
        if (s_stop) break;
    }
    if (tid == 0) {
        if (blockIdx.x == 0) {
            a.flag[0] = !s_fail && s_stop == 1;
            a.flag[1] = it;
        }
        if (s_fail) {
            set_error(a.wait.err, kErrBarrierTimeout);
            *a.wait.fail = 1;
        }
    }
}
size_t lpcg_bytes(int rounds) {
    return sizeof(LevelSmem) + sizeof(float) * 2 * kRows * kP + (size_t)rounds * (2 * sizeof(int) * kRows + sizeof(int4) + kTile);
}
using LpcgKernel = void (*)(LpcgArgs);
LpcgKernel lpcg_kernel(int rounds) { return rounds > kRun ? (LpcgKernel)k_lpcg_grid<true> : (LpcgKernel)k_lpcg_grid<false>; }
int tiles_of(const LpState& L, int* tx, int* ty) {
    *tx = (L.dims[0][0] + kTX - 1) / kTX;
    *ty = (L.dims[0][1] + kTY - 1) / kTY;
    return *tx * *ty * ((L.dims[0][2] + kTZ - 1) / kTZ);
}
}  // namespace

bool plan_lpcg_grid(const GridDev& g, const LpState& L, int sms) {
    int tx, ty;
    const int nt = tiles_of(L, &tx, &ty), rounds = (nt + sms - 1) / std::max(1, sms);
    if (L.nlev < 2 || g.nv > kLpcgMostNodes || sms < 1 || sms > kMostCtas || rounds > kMostRounds) return false;
    int n = 0;
    const auto kernel = lpcg_kernel(rounds);
    const bool ok = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)lpcg_bytes(kMostRounds)) == cudaSuccess &&
                    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, kThr, lpcg_bytes(rounds)) == cudaSuccess &&
                    n > 0;
    if (!ok) cudaGetLastError();
    return ok;
}

void launch_lpcg_grid(const GridDev& g, SolveWork& w, const LpState& L, float* d2, float* r_alt, double r2, double target_rr,
                      int cap, cudaStream_t s, int sms) {
    LpcgArgs a;
    a.g = g;
    a.f = lp_node_view(g, L, nullptr);
    a.z1 = lp_level_view(L, 1, L.z[1]);
    a.e1 = lp_level_view(L, 1, L.e[1]);
    a.e2 = L.nlev > 2 ? lp_level_view(L, 2, L.e[2]) : LView{};
    lp_build_dense(L, s);
    lp_coarse_setup(L, L.dense_level == 1 ? 1 : 2, a.z1, a.lev);
    a.lev.fold[1] = L.fold;
    a.r[0] = w.r;
    a.r[1] = r_alt;
    a.d[0] = w.d;
    a.d[1] = d2;
    a.z = w.z;
    a.q = w.q;
    a.e = w.e;
    a.kind = reinterpret_cast<const uint16_t*>(w.kind);
    a.S0 = L.W + L.lay.s0;
    a.sc = sum_scales(g, r2);
    a.target = ff_from_double(target_rr * a.sc.rr);
    a.cap = cap;
    a.ntiles = tiles_of(L, &a.tx_n, &a.ty_n);
    a.rounds = (a.ntiles + sms - 1) / sms;
    a.flag = w.flag;
    a.sync = reinterpret_cast<GridSync*>(w.gpart);
    a.wait = GridWait{&a.sync->arrived, w.wait_polls, w.err, w.flag + 2};
    cudaMemsetAsync(a.sync, 0, sizeof(unsigned), s);
    void* args[] = {&a};
    cudaLaunchCooperativeKernel((const void*)lpcg_kernel(a.rounds), dim3((unsigned)sms), dim3(kThr), args,
                                lpcg_bytes(a.rounds), s);
}
}  // namespace pic
