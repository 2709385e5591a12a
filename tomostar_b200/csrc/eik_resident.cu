// The resident solver: small grids solved by one block cluster per field, the whole field in the
// cluster's shared memory.
//
// What bounds a small job. A sweep's plane order i'+j'+k' = p is a serial chain of nx+ny+nz−2 steps,
// and a solve takes some 50 sweeps, so one field's time is the number of steps times the latency of a
// step, whatever the GPU could do beside it. The tiled engine walks that chain tile by tile (a
// 61×61×31 field: 16 tile diagonals of 44 steps and two grid-wide barriers each, 704 steps a sweep at
// about 1 µs; 57 ms in all, 9.7 as it is now); here every plane of the grid is one step: 151 steps a sweep
// at 0.4–0.7 µs, each one shared-memory update per thread and a block barrier.
//
// Layout. The (y, z) rows of the grid are dealt as a cy × cz arrangement of boxes, one per block; a
// thread owns one row along x. The block keeps its box's times with a two-node halo, one due byte per
// node in the same layout and one fixed bit per node. What a step leaves within two rows of a box face
// goes into the neighbour block's halo and due bytes (distributed shared memory stores; nothing is ever
// read remotely). Nodes of one plane are never neighbours, so no step reads what another thread writes
// in it.
//
// A box waits only for the boxes before it along the sweep, plane by plane, and not for the boxes after
// it, so the exchange costs a lag of a step or two per box and not a cluster barrier per step (measured
// on 61×61×31: 11.3 ms with a barrier per step; 7.6 with the rows' threads sending and waiting
// themselves; 5.7 with three warps of their own for it; 5.1, and 3.9 for 5.6 in fast mode, since these
// skip the planes in which nothing near a face changed, most of them after the first sweeps), and
// sweeps overlap where their orderings allow.
//
// The values are those of the tiled engine and of the reference to the bit: the same update on the
// same inputs in a plane order (SphericalEikonal.cs:297-321), the same due rule
// (EikonalOpenCl.cs:528-532, 608-622) or the fast mode's, the same round ends (:241-269).
#include <algorithm>
#include <cstring>
#include <type_traits>
#include <vector>

#include "eik_kernels.cuh"
#include "eik_resident.h"

namespace ts {
namespace eik {

namespace {

constexpr int kMaxRows = 416;  // a thread each, and three warps besides in a cluster (512 threads: 128 registers)
constexpr int kMaxCluster = 16;

struct ResGrid {
    int nx, ny, nz;
    int cy, cz;      // boxes along y and z (cy · cz <= cluster)
    int yl, zl;      // rows and levels per box (the last ones may hold fewer, at least four)
    int pitch_x;     // elements per row in shared memory: nx + 4, made even (no bank conflicts along y)
    int varz, pitch; // pitch: elements per padded row of the field in device memory
    const void *wx, *wy, *zc;
    double wz1, wz2;
};

template <typename Real>
struct ResField {
    Real* T;
    const Real* s;
    FieldState* state;
    int grid, seed_begin, seed_count, cap;
};

template <typename Real>
struct ResArgs {
    const ResGrid* grids;
    const ResField<Real>* fields;
    const int* seed_node;
    const double* seed_t;
    Control* ctl;
    const volatile int* cancel;
    int cluster, xoff;
    Real tol, wake_rel;
    int causal;
};

TS_DEVINL unsigned cluster_rank() {
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
TS_DEVINL unsigned remote_addr(unsigned local, unsigned rank) {
    unsigned a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(local), "r"(rank));
    return a;
}
TS_DEVINL void remote_store(unsigned addr, double v) {
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(addr), "d"(v) : "memory");
}
TS_DEVINL void remote_store(unsigned addr, Pair v) {
    asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(addr), "f"(v.hi), "f"(v.lo) : "memory");
}
TS_DEVINL void remote_store_u8(unsigned addr, unsigned v) {
    asm volatile("st.shared::cluster.u8 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}
TS_DEVINL void remote_store_s32(unsigned addr, int v) {
    asm volatile("st.shared::cluster.s32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}
// A neighbour's step count: stored with release after the block's own barrier, read with acquire.
TS_DEVINL void remote_publish(unsigned addr, int v) {
    asm volatile("st.release.cluster.shared::cluster.s32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}
TS_DEVINL int local_acquire(unsigned addr) {
    int v;
    asm volatile("ld.acquire.cluster.shared::cta.s32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
    return v;
}
// The box's own step count, from its first thread (after the rows' barrier) to the couriers.
TS_DEVINL void block_publish(int* at, int v) {
    asm volatile("st.release.cta.shared::cta.s32 [%0], %1;" ::"r"(unsigned(__cvta_generic_to_shared(at))), "r"(v) : "memory");
}
TS_DEVINL int block_acquire(const int* at) {
    int v;
    asm volatile("ld.acquire.cta.shared::cta.s32 %0, [%1];" : "=r"(v) : "r"(unsigned(__cvta_generic_to_shared(at))) : "memory");
    return v;
}
TS_DEVINL void rows_sync(int n) { asm volatile("bar.sync 1, %0;" ::"r"(n) : "memory"); }
constexpr int kMaxPolls = 1 << 22;  // a wait longer than about a second gives up (TS_E_TIMEOUT)
TS_DEVINL void cluster_arrive() {
    __syncwarp();  // the aligned form: the whole warp together
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}
TS_DEVINL void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

TS_HDINL size_t up16(size_t b) { return (b + 15) / 16 * 16; }
// Shared memory of a box: times, due bytes, fixed bits, and a byte per plane and pair of faces.
TS_HDINL size_t box_elems(const ResGrid& g) { return size_t(g.pitch_x) * (g.yl + 4) * (g.zl + 4); }
TS_HDINL int box_planes(const ResGrid& g) { return g.nx + g.yl + g.zl; }
TS_HDINL size_t box_bytes(const ResGrid& g) {
    const size_t elems = box_elems(g);
    return up16(8 * elems) + up16(elems) + up16((elems + 31) / 32 * 4) + up16(2 * size_t(box_planes(g)));
}

template <typename Real, bool VARZ, bool CLUSTER, int MAXT>
__global__ void __launch_bounds__(MAXT, 1) resident_kernel(ResArgs<Real> a) {
    extern __shared__ __align__(16) unsigned char smem[];
    // Every box's word at a round's end, in two turns: a block without a box waits for no neighbour, so the words
    // of the next round may come before it has read these; the round after that waits for it.
    __shared__ int flags[2][kMaxCluster];
    __shared__ int done_here;   // steps finished by this box
    __shared__ int done_by[4];  // steps finished by the neighbour box at y−1, y+1, z−1, z+1
    const int rank = CLUSTER ? int(cluster_rank()) : 0;
    const ResField<Real>& fd = a.fields[CLUSTER ? blockIdx.x / a.cluster : blockIdx.x];
    const ResGrid g = a.grids[fd.grid];
    const int nx = g.nx, X = g.pitch_x, XY = X * (g.yl + 4);
    const size_t elems = box_elems(g);
    Real* T = reinterpret_cast<Real*>(smem);
    uint8_t* due = smem + up16(8 * elems);
    uint32_t* fixed = reinterpret_cast<uint32_t*>(due + up16(elems));
    // Per plane of the box: a row near the y faces, near the z faces changed in it.
    const int planes_max = box_planes(g);
    uint8_t* moved = reinterpret_cast<uint8_t*>(fixed) + up16((elems + 31) / 32 * 4);
    const unsigned T_s = unsigned(__cvta_generic_to_shared(T)), due_s = unsigned(__cvta_generic_to_shared(due)),
                   flags_s = unsigned(__cvta_generic_to_shared(&flags[0][0])),
                   done_s = unsigned(__cvta_generic_to_shared(done_by));
    const int by = rank % g.cy, bz = rank / g.cy;
    const bool idle = bz >= g.cz;  // a block the arrangement has no box for
    const int j0 = by * g.yl, k0 = bz * g.zl;
    const int nyl = idle ? 0 : min(g.yl, g.ny - j0), nzl = idle ? 0 : min(g.zl, g.nz - k0);
    // In a cluster three more warps carry the exchange, so that the rows' threads run nothing of it: one
    // watches the boxes before this one and holds back the step's barrier, two copy what the step wrote
    // near the y and z faces to the neighbours and tell them how far this box is.
    const int tid = threadIdx.x, nt = CLUSTER ? blockDim.x - 96 : blockDim.x;
    const bool watcher = CLUSTER && tid >= nt && tid < nt + 32, courier = CLUSTER && tid >= nt + 32;
    const Real inf = real_inf<Real>();

    if (tid < 4) done_by[tid] = 0;
    if (tid == 0) done_here = 0;
    for (int q = tid; q < 2 * planes_max && CLUSTER; q += blockDim.x) moved[q] = 0;
    // +inf everywhere, every node of the box due, the seeds (own and halo) in place.
    for (size_t q = tid; q < elems; q += blockDim.x) {
        T[q] = inf;
        due[q] = 0;
    }
    for (size_t q = tid; q < (elems + 31) / 32; q += blockDim.x) fixed[q] = 0u;
    __syncthreads();
    const bool has_row = tid < nyl * nzl && tid < nt;
    const int jl = has_row ? tid % nyl : 0, kl = has_row ? tid / nyl : 0;
    const int j = j0 + jl, k = k0 + kl;
    const int row = (kl + 2) * XY + (jl + 2) * X + 2;  // element of the row's node i = 0
    if (has_row)
        for (int i = 0; i < nx; i++) due[row + i] = 1;
    for (int q = tid; q < fd.seed_count && !idle; q += blockDim.x) {
        const int node = __ldg(&a.seed_node[fd.seed_begin + q]);
        const int si = node % nx, r = node / nx, sj = r % g.ny - j0, sk = r / g.ny - k0;
        if (sj < -2 || sj >= nyl + 2 || sk < -2 || sk >= nzl + 2) continue;
        const int c = (sk + 2) * XY + (sj + 2) * X + 2 + si;
        T[c] = Real(a.seed_t[fd.seed_begin + q]);
        if (sj >= 0 && sj < nyl && sk >= 0 && sk < nzl) atomicOr(&fixed[c >> 5], 1u << (c & 31));
    }
    __syncthreads();
    // The part of the row that holds fixed nodes (empty for most rows): only there is the bit looked up.
    int fx_lo = 0, fx_len = 0;
    if (has_row) {
        int lo = nx, hi = -1;
        for (int i = 0; i < nx; i++)
            if ((fixed[(row + i) >> 5] >> ((row + i) & 31)) & 1u) {
                lo = min(lo, i);
                hi = i;
            }
        if (hi >= 0) {
            fx_lo = lo;
            fx_len = hi - lo + 1;
        }
    }
    // The row's weights and slowness; the neighbours' boxes that its changes reach.
    const int64_t rowi = int64_t(k) * g.ny + j;
    Real wx1 = Real(1), wx2 = Real(1), wy1 = Real(1), wy2 = Real(1);
    if (has_row) {
        const Real* wx = static_cast<const Real*>(g.wx);
        const Real* wy = static_cast<const Real*>(g.wy);
        wx1 = ldg_r(&wx[2 * rowi]);
        wx2 = ldg_r(&wx[2 * rowi + 1]);
        wy1 = ldg_r(&wy[2 * k]);
        wy2 = ldg_r(&wy[2 * k + 1]);
    }
    const Real wz1 = Real(g.wz1), wz2 = Real(g.wz2);
    const Real* zc = VARZ && g.varz ? static_cast<const Real*>(g.zc) + kZCoef * k : nullptr;
    const Real* __restrict__ srow = fd.s + rowi * nx;
    // A courier's faces: along its axis the box before (side 0) and after (side 1), the elements from one row
    // to the next, where this box's elements lie in the neighbour's arrays (all boxes but the last hold yl
    // rows and zl levels, so the shift is the same from both sides), and its slots of the step counts.
    const bool cz_ = courier && tid >= nt + 64;
    const int c_st = cz_ ? XY : X, c_n = cz_ ? nzl : nyl, c_m = cz_ ? nyl : nzl;
    const int c_box = (cz_ ? g.zl : g.yl) * c_st, c_rank = cz_ ? g.cy : 1;
    uint8_t* const c_moved = moved + (cz_ ? planes_max : 0);
    // Rows whose changes a courier has to carry.
    const bool ye = CLUSTER && has_row && ((jl < 2 && by > 0) || (jl >= nyl - 2 && by + 1 < g.cy));
    const bool ze = CLUSTER && has_row && ((kl < 2 && bz > 0) || (kl >= nzl - 2 && bz + 1 < g.cz));
    const bool c_on[2] = {courier && !idle && (cz_ ? bz > 0 : by > 0), courier && !idle && (cz_ ? bz + 1 < g.cz : by + 1 < g.cy)};
    if (CLUSTER) {
        cluster_arrive();  // every box is in place before a neighbour writes into it
        cluster_wait();
    }

    const int planes = nx + g.ny + g.nz - 2;
    const Real tol = a.tol, wake_rel = a.wake_rel, none = minus_inf<Real>();
    const bool causal = a.causal != 0;
    unsigned long long evals = 0;
    int phase = 0, round = 0, rounds0 = 0, rounds1 = 0, status = kRunning;
    int base = 0;  // steps of the sweeps before this one
    int turn = 0;  // of the flags
    bool cancelled = false, dead = false;
    while (status == kRunning) {
        bool big = false;
        for (int dir = 0; dir < 8; dir++, base += planes) {
            const bool mx = dir & 1, my = dir & 2, mz = dir & 4;
            // A row's node of plane p is i' = p − off, off its canonical j' + k'; the box's rows hold nodes
            // of the planes [p0, p1).
            auto off_of = [&](int rj, int rk) { return (my ? g.ny - 1 - rj : rj) + (mz ? g.nz - 1 - rk : rk); };
            const int p0 = idle ? 0 : off_of(my ? j0 + nyl - 1 : j0, mz ? k0 + nzl - 1 : k0);
            const int p1 = idle ? 0 : p0 + nx + nyl + nzl - 2;
            if (CLUSTER && watcher) {
                // Step p starts when the boxes before this one along the sweep have finished plane p − 1.
                const bool upy = !idle && (my ? by + 1 < g.cy : by > 0), dny = !idle && (my ? by > 0 : by + 1 < g.cy);
                const bool upz = !idle && (mz ? bz + 1 < g.cz : bz > 0), dnz = !idle && (mz ? bz > 0 : bz + 1 < g.cz);
                const unsigned upy_s = done_s + (my ? 4 : 0), upz_s = done_s + (mz ? 12 : 8);
                const unsigned dny_s = done_s + (my ? 0 : 4), dnz_s = done_s + (mz ? 8 : 12);
                // A sweep starts as the box finishes the one before. Along an axis that has not turned round
                // the box after this one lags: it must have finished that sweep, whose values this one reads.
                // (Along one that has, it was before this box, which has waited for all that it reads.)
                const int turned = dir ^ ((dir + 7) & 7);
                const bool wait_y = dny && !(turned & 2), wait_z = dnz && !(turned & 4);
                int seen_y = upy ? 0 : 1 << 30, seen_z = upz ? 0 : 1 << 30;
                for (int p = p0; p <= p1; p++) {
                    int polls = 0;
                    const int need = p < p1 ? base + p : 0;  // the sweep's last barrier waits for nothing
                    if (!dead) {
                        if (p == p0) {
                            while (wait_y && local_acquire(dny_s) < base && polls < kMaxPolls) polls++;
                            while (wait_z && local_acquire(dnz_s) < base && polls < kMaxPolls) polls++;
                        }
                        for (; seen_y < need && polls < kMaxPolls; polls++) seen_y = local_acquire(upy_s);
                        for (; seen_z < need && polls < kMaxPolls; polls++) seen_z = local_acquire(upz_s);
                        dead = polls >= kMaxPolls;
                    }
                    rows_sync(nt + 32);
                }
            } else if (CLUSTER && courier) {
                int told = base + p0;
                auto tell = [&](int done) {
                    __syncwarp();
                    if ((tid & 31) < 2 && c_on[tid & 1]) {
                        // This box is the one before (slot 0 or 2) of the one after it, and the other way.
                        const int to = (tid & 1) ? rank + c_rank : rank - c_rank;
                        remote_publish(remote_addr(done_s + (cz_ ? 8 : 0) + ((tid & 1) ? 0 : 4), to), done);
                    }
                };
                tell(told);
                while (told < base + p1) {
                    int now = told, polls = 0;
                    while (now <= told && polls < kMaxPolls) {
                        now = __shfl_sync(0xffffffffu, block_acquire(&done_here), 0);  // one value for the warp
                        polls++;
                    }
                    if (polls >= kMaxPolls) {
                        dead = true;
                        break;
                    }
                    // The nodes of the finished planes in the two rows at each face, where any changed: their
                    // times, and the due bytes of the neighbour's rows that they may have woken (set in this
                    // box's halo).
                    for (int q0 = told - base; q0 < now - base; q0 += 32) {
                        const int mine = q0 + (tid & 31);
                        const bool has = mine < now - base && *(volatile uint8_t*)&c_moved[mine - p0] != 0;
                        if (has) c_moved[mine - p0] = 0;
                        for (unsigned todo = __ballot_sync(0xffffffffu, has); todo; todo &= todo - 1) {
                            const int p = q0 + __ffs(todo) - 1;
                            for (int q = tid & 31; q < 4 * c_m; q += 32) {
                                const int side = (q >> 1) & 1, r = q & 1, m = q >> 2;
                                if (!c_on[side]) continue;
                                const int n = side ? c_n - 1 - r : r;
                                const int rj = cz_ ? m : n, rk = cz_ ? n : m;
                                const int ip = p - off_of(j0 + rj, k0 + rk);
                                if (unsigned(ip) >= unsigned(nx)) continue;
                                const int c = (rk + 2) * XY + (rj + 2) * X + 2 + (mx ? nx - 1 - ip : ip);
                                const int st = side ? c_st : -c_st, to = side ? rank + c_rank : rank - c_rank;
                                const int cn = side ? c - c_box : c + c_box;
                                remote_store(remote_addr(T_s + 8 * cn, to), T[c]);
                                if (due[c + 2 * st]) {
                                    due[c + 2 * st] = 0;
                                    remote_store_u8(remote_addr(due_s + cn + 2 * st, to), 1);
                                }
                                if (r == 0 && due[c + st]) {
                                    due[c + st] = 0;
                                    remote_store_u8(remote_addr(due_s + cn + st, to), 1);
                                }
                            }
                        }
                    }
                    told = now;
                    tell(told == base + p1 ? base + planes : told);
                }
            } else {
                const int off = has_row ? off_of(j, k) : planes;
                const int di = mx ? -1 : 1;
                int i = mx ? nx - 1 + off - p0 : p0 - off;  // the node of plane p0 (off the row until p = off)
                // The thread's node of the plane and what lies at it move one node per plane.
                Real* c = T + row + i;
                uint8_t* d = due + row + i;
                const Real* sp = srow + i;
                Real s = unsigned(i) < unsigned(nx) ? ldg_r(sp) : Real(0);
                if (CLUSTER) rows_sync(nt + 32);
                for (int p = p0; p < p1; p++) {
                    if (unsigned(i) < unsigned(nx) && *(volatile uint8_t*)d &&
                        !(unsigned(i - fx_lo) < unsigned(fx_len) && ((fixed[(row + i) >> 5] >> ((row + i) & 31)) & 1u))) {
                        *d = 0;
                        evals++;
                        const Real cur = c[0];
                        const Real xm = c[-1], xp = c[1], xm2 = c[-2], xp2 = c[2];
                        const Real ym = c[-X], yp = c[X], ym2 = c[-2 * X], yp2 = c[2 * X];
                        const Real zm = c[-XY], zp = c[XY], zm2 = c[-2 * XY], zp2 = c[2 * XY];
                        Real cand;
                        if (VARZ && g.varz)
                            cand = Update<Real, VARZ>::eval(s, xm, xp, xm2, xp2, ym, yp, ym2, yp2, zm, zp, zm2, zp2, wx1,
                                                            wx2, wy1, wy2, wz1, wz2, zc, phase == 1);
                        else
                            cand = Update<Real, false>::eval(s, xm, xp, xm2, xp2, ym, yp, ym2, yp2, zm, zp, zm2, zp2, wx1,
                                                             wx2, wy1, wy2, wz1, wz2, nullptr, phase == 1);
                        if (cand < cur) {
                            c[0] = cand;
                            if (CLUSTER && ye) moved[p - p0] = 1;
                            if (CLUSTER && ze) moved[planes_max + p - p0] = 1;
                            if (counts_as_change<Real>(cur, cand, tol)) big = true;
                            if (wakes<Real>(cur, cand, wake_rel)) {
                                // The neighbours holding more than the new time (causal rule), or all. The due
                                // bytes outside the grid exist (halo) and are never looked at.
                                const Real over = causal ? cand : none;
                                if (over < xm) d[-1] = 1;
                                if (over < xp) d[1] = 1;
                                if (over < xm2) d[-2] = 1;
                                if (over < xp2) d[2] = 1;
                                if (over < ym) d[-X] = 1;
                                if (over < yp) d[X] = 1;
                                if (over < ym2) d[-2 * X] = 1;
                                if (over < yp2) d[2 * X] = 1;
                                if (over < zm) d[-XY] = 1;
                                if (over < zp) d[XY] = 1;
                                if (over < zm2) d[-2 * XY] = 1;
                                if (over < zp2) d[2 * XY] = 1;
                            }
                        }
                    }
                    i += di;  // the next plane's slowness is on its way while the others arrive
                    c += di;
                    d += di;
                    sp += di;
                    s = unsigned(i) < unsigned(nx) ? ldg_r(sp) : Real(0);
                    if (CLUSTER) {
                        rows_sync(nt + 32);
                        if (tid == 0) block_publish(&done_here, base + p + 1);
                    } else {
                        __syncthreads();
                    }
                }
            }
            if (CLUSTER) __syncthreads();  // the couriers have sent this sweep's values before the next changes them
        }
        // Round end (SphericalEikonal.cs:297-323; EikonalOpenCl.cs:241-269): every block takes the same
        // decision from the cluster's flags (bit 0: something changed, bit 1: cancelled).
        // bit 2: a wait ran out.
        int mine = (tid == 0 && rank == 0 && a.cancel && *a.cancel) ? 2 : 0;
        mine = (__syncthreads_or(big) ? 1 : 0) | (__syncthreads_or(mine) ? 2 : 0) | (__syncthreads_or(dead) ? 4 : 0);
        if (CLUSTER) {
            if (tid < a.cluster) remote_store_s32(remote_addr(flags_s + 4 * (turn * kMaxCluster + rank), tid), mine);
            cluster_arrive();
            cluster_wait();
            mine = 0;
            for (int q = 0; q < a.cluster; q++) mine |= flags[turn][q];
            turn ^= 1;
        }
        if (mine & 4) {
            dead = true;
            break;
        }
        cancelled = (mine & 2) != 0;
        if (!(mine & 1)) {
            if (phase == 0) {
                rounds0 = round + 1;
                phase = 1;
                round = 0;
                // Phase 1 starts with every node due (EikonalOpenCl.cs:235-239); the next step's barrier
                // is not needed before it, since a node's own thread alone reads its due byte first.
                if (has_row)
                    for (int q = 0; q < nx; q++) due[row + q] = 1;
                if (CLUSTER) {
                    cluster_arrive();
                    cluster_wait();
                } else {
                    __syncthreads();
                }
            } else {
                rounds1 = round + 1;
                status = kSettled;
            }
        } else {
            round++;
            if (round >= fd.cap) {
                if (phase == 0) rounds0 = round;
                else rounds1 = round;
                status = kUnsettled;
            }
        }
        if (cancelled) break;
    }
    // The field to device memory (a warp per row).
    const int warp = tid >> 5, lane = tid & 31;
    for (int r = warp; r < nyl * nzl; r += blockDim.x >> 5) {
        const int rj = r % nyl, rk = r / nyl;
        const Real* src = T + (rk + 2) * XY + (rj + 2) * X + 2;
        Real* dst = fd.T + (int64_t(k0 + rk) * g.ny + j0 + rj) * g.pitch + a.xoff;
        for (int q = lane; q < nx; q += 32) dst[q] = src[q];
    }
    for (int o = 16; o > 0; o >>= 1) evals += __shfl_down_sync(0xffffffffu, evals, o);
    if (lane == 0 && evals) atomicAdd(&a.ctl->updates, evals);
    if (tid == 0) {
        atomicAdd(&a.ctl->visits, 8ull * (unsigned long long)(rounds0 + rounds1));
        if (rank == 0) {
            fd.state->status = status;
            fd.state->rounds0 = rounds0;
            fd.state->rounds1 = rounds1;
            if (dead) atomicCAS(&a.ctl->error, 0, TS_E_TIMEOUT);
            if (cancelled && status == kRunning) atomicCAS(&a.ctl->error, 0, TS_E_CANCELLED);
        }
    }
}

// The arrangement of a grid's rows over at most `cluster` boxes: the one with the fewest rows per box
// whose boxes fit in shared memory, at least four rows and levels in every box of a divided axis. False: none.
bool arrange(const host::Grid& g, int cluster, size_t smem_max, ResGrid& out) {
    int best_rows = 1 << 30;
    size_t best_bytes = 0;
    for (int cz = 1; cz <= cluster; cz++)
        for (int cy = 1; cy * cz <= cluster; cy++) {
            ResGrid t{};
            t.nx = g.nx;
            t.yl = (g.ny + cy - 1) / cy;
            t.zl = (g.nz + cz - 1) / cz;
            // As many boxes as the rows fill, the last with at least four.
            t.cy = (g.ny + t.yl - 1) / t.yl;
            t.cz = (g.nz + t.zl - 1) / t.zl;
            if ((t.cy > 1 && (t.yl < 4 || g.ny - (t.cy - 1) * t.yl < 4)) ||
                (t.cz > 1 && (t.zl < 4 || g.nz - (t.cz - 1) * t.zl < 4)))
                continue;
            t.pitch_x = (g.nx + 5) / 2 * 2;
            const int rows = t.yl * t.zl;
            const size_t bytes = box_bytes(t);
            if (rows > kMaxRows || bytes > smem_max) continue;
            if (rows < best_rows || (rows == best_rows && bytes < best_bytes)) {
                best_rows = rows;
                best_bytes = bytes;
                out = t;
            }
        }
    out.ny = g.ny;
    out.nz = g.nz;
    out.varz = g.variable ? 1 : 0;
    return best_rows < (1 << 30);
}

constexpr size_t kSmemMax = 226 * 1024;

}  // namespace

// The rule. A solve's time here is its chain of steps whatever the cluster size, within 20 % (40×40×20,
// one field: 5.0, 4.8, 4.0 and 4.2 ms with 2, 4, 8 and 16 blocks), so the size is the smallest that
// holds every grid, or up to eight blocks where the fields still run in as many waves: a cluster lies in
// one GPC, which takes 16 / C clusters. One wave takes half of the tiled engine's time (61×61×31, one
// field: 5.1 ms against 9.7; 40×40×20, 54 fields: 6.3 against 9.1; 48×48×24, 18: 7.1 against 11.3), and the
// engine's grows slowly with the fields, so more are the engine's (61×61×31, 18 fields: 18.5 against 15.6;
// 70×70×35, 16: 22.8 against 18.4; 48×48×24, 54: 13.3 against 11.7), but for a few over a wave (61×61×31,
// 9 fields: 11.5 against 15.1; 48×48×24, 36: 11.0 against 11.4). Grids that one block holds: up to two
// waves (22×20×16, 148 fields: 2.0 against 4.0; 296: 3.7 against 4.1; 440: 5.1 against 5.2).
int resident_cluster(ts_ctx* ctx, const EngineJob& job) {
    if (job.fields.empty()) return 0;
    const int gpcs = std::max(1, ctx->sm_count / 18);
    const int nf = int(job.fields.size());
    auto at_once = [&](int c) { return c == 1 ? ctx->sm_count : gpcs * (kMaxCluster / c); };
    auto waves = [&](int c) { return (nf + at_once(c) - 1) / at_once(c); };
    auto fits = [&](int c) {
        for (auto* g : job.grids) {
            ResGrid t{};
            if (!arrange(*g, c, kSmemMax, t)) return false;
        }
        return true;
    };
    int c = 1;
    while (c <= kMaxCluster && !fits(c)) c *= 2;
    if (c > kMaxCluster || nf > (c == 1 ? 2 * at_once(c) : at_once(c) + at_once(c) / 8)) return 0;
    if (c == 1) return 1;  // no exchange at all
    while (c < 8 && waves(2 * c) == waves(c)) c *= 2;
    return c;
}

template <typename Real>
std::optional<int> resident_run(ts_ctx* ctx, EngineJob& job, int cluster, ts_eik_stats* stats, cudaStream_t s) {
    const int nf = int(job.fields.size()), ng = int(job.grids.size());
    // One image of everything the launch reads: grids, weights, fields, seeds, control, states.
    std::vector<uint8_t> h;
    auto add = [&](size_t bytes) {
        const size_t off = (h.size() + 15) / 16 * 16;
        h.resize(off + std::max<size_t>(bytes, 1), 0);
        return off;
    };
    const size_t o_grids = add(sizeof(ResGrid) * ng), o_fields = add(sizeof(ResField<Real>) * nf),
                 o_ctl = add(sizeof(Control)), o_states = add(sizeof(FieldState) * nf);
    std::vector<ResGrid> grids(ng);
    std::vector<size_t> o_wx(ng), o_wy(ng), o_zc(ng);
    size_t smem = 0;
    int threads = 32;
    bool any_var = false;
    for (int q = 0; q < ng; q++) {
        const host::Metric& m = *job.metrics[q];
        if (!arrange(*job.grids[q], cluster, kSmemMax, grids[q])) return ctx->fail(TS_E_ARG, "grid too large");
        grids[q].pitch = job.pitch[q];
        grids[q].wz1 = weight_of<Real>(m.wz1, m.wz1_32);
        grids[q].wz2 = weight_of<Real>(m.wz2, m.wz2_32);
        smem = std::max(smem, box_bytes(grids[q]));
        threads = std::max(threads, (grids[q].yl * grids[q].zl + 31) / 32 * 32);
        any_var |= grids[q].varz != 0;
        o_wx[q] = add(sizeof(Real) * m.wx.size());
        for (size_t e = 0; e < m.wx.size(); e++)
            reinterpret_cast<Real*>(h.data() + o_wx[q])[e] = Real(weight_of<Real>(m.wx[e], m.wx32[e]));
        o_wy[q] = add(sizeof(Real) * m.wy.size());
        for (size_t e = 0; e < m.wy.size(); e++)
            reinterpret_cast<Real*>(h.data() + o_wy[q])[e] = Real(weight_of<Real>(m.wy[e], m.wy32[e]));
        o_zc[q] = add(sizeof(Real) * m.zc.size());
        for (size_t e = 0; e < m.zc.size(); e++) reinterpret_cast<Real*>(h.data() + o_zc[q])[e] = Real(m.zc[e]);
    }
    size_t seeds = 0;
    for (auto& f : job.fields) seeds += f.seed_idx.size();
    const size_t o_node = add(4 * seeds), o_t = add(8 * seeds);
    uint8_t* D = static_cast<uint8_t*>(ctx->buf("res.arena", h.size()));
    uint8_t* image = static_cast<uint8_t*>(ctx->host_buf("res.arena.image", h.size()));
    const size_t back = sizeof(FieldState) * nf + (o_states - o_ctl);  // control and states, one copy
    uint8_t* res_h = static_cast<uint8_t*>(ctx->host_buf("res.back", back));
    if (!D || !image || !res_h) return TS_E_NOMEM;
    for (int q = 0; q < ng; q++) {
        grids[q].wx = D + o_wx[q];
        grids[q].wy = D + o_wy[q];
        grids[q].zc = D + o_zc[q];
        std::memcpy(h.data() + o_grids + sizeof(ResGrid) * q, &grids[q], sizeof(ResGrid));
    }
    size_t at = 0;
    for (int f = 0; f < nf; f++) {
        const EngineField& ef = job.fields[f];
        ResField<Real> rf{};
        rf.T = static_cast<Real*>(ef.T);
        rf.s = static_cast<const Real*>(ef.slowness);
        rf.state = reinterpret_cast<FieldState*>(D + o_states) + f;
        rf.grid = ef.grid;
        rf.seed_begin = int(at);
        rf.seed_count = int(ef.seed_idx.size());
        rf.cap = ef.cap;
        std::memcpy(h.data() + o_fields + sizeof rf * f, &rf, sizeof rf);
        std::memcpy(h.data() + o_node + 4 * at, ef.seed_idx.data(), 4 * ef.seed_idx.size());
        std::memcpy(h.data() + o_t + 8 * at, ef.seed_t.data(), 8 * ef.seed_t.size());
        at += ef.seed_idx.size();
    }
    std::memcpy(image, h.data(), h.size());
    ResArgs<Real> args{};
    args.grids = reinterpret_cast<const ResGrid*>(D + o_grids);
    args.fields = reinterpret_cast<const ResField<Real>*>(D + o_fields);
    args.seed_node = reinterpret_cast<const int*>(D + o_node);
    args.seed_t = reinterpret_cast<const double*>(D + o_t);
    args.ctl = reinterpret_cast<Control*>(D + o_ctl);
    args.cancel = ctx->cancel_dev;
    args.cluster = cluster;
    args.xoff = job.xoff;
    args.tol = Real(job.tol);
    args.wake_rel = Real(job.wake_rel);
    args.causal = job.wake_rel > 0 ? 1 : 0;
    // Up to 256 rows a block leave room for all of a thread's registers.
    auto pick = [&](auto maxt) {
        constexpr int T = decltype(maxt)::value;
        return cluster > 1 ? (any_var ? resident_kernel<Real, true, true, T> : resident_kernel<Real, false, true, T>)
                           : (any_var ? resident_kernel<Real, true, false, T> : resident_kernel<Real, false, false, T>);
    };
    const int max_threads = threads <= 256 ? 352 : 512;
    auto kfn = threads <= 256 ? pick(std::integral_constant<int, 352>()) : pick(std::integral_constant<int, 512>());
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(unsigned(nf) * cluster);
    cfg.blockDim = dim3(threads + (cluster > 1 ? 96 : 0));
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = cluster;
    attr.val.clusterDim.y = 1;
    attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = cluster > 1 ? 1 : 0;
    // A device that cannot place such a cluster (a part of a GPU, GPCs with few SMs) leaves the job to the engine. Asked
    // once for a kernel and size, with the most shared memory and threads that a job may want (a query takes 0.1 ms).
    auto placed = [&] {
        const auto key = std::make_pair(reinterpret_cast<const void*>(kfn), cluster);
        const auto known = ctx->clusters_placed.find(key);
        if (known != ctx->clusters_placed.end()) return known->second;
        cudaLaunchConfig_t most = cfg;
        most.blockDim = dim3(max_threads);
        most.dynamicSmemBytes = kSmemMax;
        int at_once = 0;
        const bool yes =
            cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kSmemMax)) == cudaSuccess &&
            (cluster <= 8 || cudaFuncSetAttribute(kfn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess) &&
            cudaOccupancyMaxActiveClusters(&at_once, kfn, &most) == cudaSuccess && at_once > 0;
        ctx->clusters_placed[key] = yes;
        return yes;
    };
    auto takes = [&] {
        return (cluster == 1 || placed()) &&
               cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem)) == cudaSuccess;
    };
    if (!takes()) {
        cudaGetLastError();
        return std::nullopt;
    }
    EventPair ev;
    TS_CUDA_TRY(ctx, cudaMemcpyAsync(D, image, h.size(), cudaMemcpyHostToDevice, s));
    cudaEventRecord(ev.a, s);
    if (cudaLaunchKernelEx(&cfg, kfn, args) != cudaSuccess) {
        cudaGetLastError();
        return std::nullopt;
    }
    cudaEventRecord(ev.b, s);
    TS_CUDA_TRY(ctx, cudaMemcpyAsync(res_h, D + o_ctl, back, cudaMemcpyDeviceToHost, s));
    TS_CUDA_TRY(ctx, cudaStreamSynchronize(s));
    float kms = 0;
    cudaEventElapsedTime(&kms, ev.a, ev.b);
    const Control ctl = *reinterpret_cast<const Control*>(res_h);
    const FieldState* st = reinterpret_cast<const FieldState*>(res_h + (o_states - o_ctl));
    if (stats) {
        stats->kernel_ms += kms;
        stats->node_updates += int64_t(ctl.updates);
        stats->tile_visits += int64_t(ctl.visits);
        stats->launches += 1;
    }
    for (int f = 0; f < nf; f++) {
        job.fields[f].initialized = true;
        job.fields[f].status = st[f].status;
        job.fields[f].rounds[0] = st[f].rounds0;
        job.fields[f].rounds[1] = st[f].rounds1;
    }
    if (ctl.error == TS_E_CANCELLED) return ctx->fail(TS_E_CANCELLED, "cancelled");
    if (ctl.error) return ctx->fail(ctl.error, "resident solver: a device-side wait ran out");
    return TS_OK;
}

template std::optional<int> resident_run<double>(ts_ctx*, EngineJob&, int, ts_eik_stats*, cudaStream_t);
template std::optional<int> resident_run<Pair>(ts_ctx*, EngineJob&, int, ts_eik_stats*, cudaStream_t);

}  // namespace eik
}  // namespace ts
