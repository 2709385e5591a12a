// The block tile of the engine: 32×BY×BZ nodes swept by one thread block with one thread per (y, z) row.
//
// What bounds a sweep is the latency of its steps and the instructions of a step, not bandwidth (24 B of
// the 8-byte values per update, 69 B of DRAM traffic, a seventh of the copy rate). The warp-sized
// tiles this replaces (32×8×4 rows in registers, neighbours by shuffles) spent 757 warp instructions on a
// step of up to 32 updates, of which the update is some 220, and crossed a 121×121×61 field in 34
// diagonals of 44 steps. Here the tile and its two-node halo lie in shared memory in grid orientation, so
// a step is 13 loads at fixed offsets from one address, the update, one store and a byte per woken node;
// the field is crossed in 18 diagonals of 54 steps. Measured against the better of the earlier shapes (kernel
// time, both by diagonals, in turn on one GPU): 50 fields of 121×121×61 162 -> 56 ms, 24 of 401×401×121
// 1,205 -> 673, 400 of 101×101×61 341 -> 244. Since tiles start as their neighbours allow (eik_flow.cuh), all on
// one GPU: 50 of 121×121×61 49 ms, 10 of 161×161×81 (every drop wakes) 82, 25 of 81×81×41 19, 24 of 401×401×121
// 733, 16 uneven grids in FP32 27. A plane with due nodes takes some 1,500 cycles, 850 of them the update's
// chain; a visit's load, write-back and tokens some 20,000.
//
// Inside a tile the reference's plane order i'+j'+k' = p (mirrored coordinates) is kept: at step p the
// thread of canonical row (j', k') evaluates the node i' = p − j' − k', one block barrier per step. A
// node's neighbours lie on other planes, so a step reads nothing that another thread writes in it.
// (Warps that wait only for the warps before them instead of a barrier took 15 to 20 % longer: the
// hand-over costs more than the barrier where most planes hold due nodes.)
//
// Due nodes are tracked per node as the reference's dirty flags (EikonalOpenCl.cs:528-532, 608-622):
// a byte per node of the tile and its halo during a visit (a wake is a plain store; atomics on bit words
// took 10 % longer), a bit per node between visits; the halo's go to the neighbour tiles at the end.
#pragma once

#include "eik_flow.cuh"

namespace ts {
namespace eik {

template <typename Real, int BX, int BY, int BZ>
struct BlockTile {
    static_assert(BX == 32 && sizeof(Real) == 8 && BY % 8 == 0 && BZ % 4 == 0, "rows of 32 nodes, warps of 8x4 rows");
    static constexpr int kThreads = BY * BZ;
    static constexpr int HX = Layout<Real>::HX;
    static constexpr int PITCH = BX + 2 * HX;         // values per row, x halo included
    static constexpr int RY = BY + 4, RZ = BZ + 4;    // rows and levels, halo included
    static constexpr int LEVEL = RY * PITCH;
    static constexpr int kSlots = RY * RZ;            // row (j, k) is slot (k + 2)·RY + j + 2
    // The first and the last two slots are corners, which nothing reads: they are not stored.
    static constexpr int kTimeBytes = (kSlots - 4) * PITCH * 8;
    // Due bytes: row r's node i is byte r·DP + 4 + i. The two bytes before a row's first node and the two
    // after its last (the first two of the next row's 36) are its x halo.
    static constexpr int DP = BX + 4;
    static constexpr int kDueBytes = (kSlots * DP + 4 + 15) / 16 * 16;
    static constexpr int kBytes = kTimeBytes + kDueBytes + 64;
    static constexpr int NSTEPS = BX + BY + BZ - 2;
    static constexpr int MW = BY * BZ;                // due words per tile, one per row
};

constexpr int kMaxRowWaits = 1 << 20;

struct BlockShared {  // the last 64 bytes of the block's shared memory
    unsigned long long entry;
    unsigned long long arrived;  // mbarrier of the tile's row copies
    int first[8];  // per warp: the first plane with a due node
};

// Bulk copies of whole rows (a row and its x halo in, a row out): one instruction per row where 16-byte
// asynchronous copies took one per chunk and its address arithmetic, and warps wrote rows one after
// another (50 fields of 121×121×61: 71 -> 68 ms). Every row starts on a 16-byte boundary on both sides.
TS_DEVINL unsigned smem_addr(const void* p) { return unsigned(__cvta_generic_to_shared(p)); }
TS_DEVINL void rows_expect(unsigned bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
TS_DEVINL void row_in(unsigned dst, const void* src, unsigned bytes, unsigned bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                 "l"(__cvta_generic_to_global(src)), "r"(bytes), "r"(bar)
                 : "memory");
}
TS_DEVINL void row_out(void* dst, unsigned src, unsigned bytes) {
    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(__cvta_generic_to_global(dst)),
                 "r"(src), "r"(bytes)
                 : "memory");
}
TS_DEVINL bool rows_arrived(unsigned bar, unsigned parity) {
    unsigned ok;
    asm volatile("{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}"
                 : "=r"(ok)
                 : "r"(bar), "r"(parity)
                 : "memory");
    return ok != 0;
}

// Visits one tile of one field for its sweep ordering; the whole block. Returns the thread's node
// evaluations.
template <typename Real, int BX, int BY, int BZ, bool VARZ>
TS_DEVINL int visit_block(const Args<Real>& a, const FieldDesc<Real>& fd, const TileItem& it, unsigned char* smem,
                          BlockShared* sh, unsigned parity) {
    const GridDesc& g = fd.g;
    const int tx = it.tx, ty = it.ty, tz = it.tz, dir = it.dir;
    const bool second = it.phase == 1;
    using B = BlockTile<Real, BX, BY, BZ>;
    constexpr int P = B::PITCH, L = B::LEVEL, RY = B::RY;
    Real* const T = reinterpret_cast<Real*>(smem) - 2 * P;
    uint8_t* const due = smem + B::kTimeBytes;
    constexpr int DP = B::DP, DL = RY * DP;
    const Real inf = real_inf<Real>();
    const int nx = g.nx, ny = g.ny, nz = g.nz;
    const int x0 = tx * BX, y0 = ty * BY, z0 = tz * BZ;
    const int tid = (tz * g.ty + ty) * g.tx + tx;
    const bool mx = (dir & 1) != 0, my = (dir & 2) != 0, mz = (dir & 4) != 0;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int j = (warp % (BY / 8)) * 8 + (lane & 7), k = (warp / (BY / 8)) * 4 + (lane >> 3);
    const int gy = y0 + j, gz = z0 + k;
    const bool row_on = gy < ny && gz < nz;
    const int64_t rowi = row_on ? int64_t(gz) * ny + gy : 0;
    const int slot = (k + 2) * RY + j + 2;
    const int pitch = g.pitch;

    // The tile's rows and its y and z halo rows with their x halo (the pads of a field row hold +inf, so x
    // needs no check): a thread copies its own row and one of the halo rows; +inf for rows off the grid.
    {
        const unsigned bar = smem_addr(&sh->arrived);
        const bool has_halo = t < 4 * (BY + BZ);
        int hj = 0, hk = 0;
        if (t < 4 * BZ) {
            hk = t >> 2;
            hj = (t & 3) < 2 ? (t & 3) - 2 : BY + (t & 3) - 2;
        } else if (has_halo) {
            const int h = t - 4 * BZ;
            hj = h >> 2;
            hk = (h & 3) < 2 ? (h & 3) - 2 : BZ + (h & 3) - 2;
        }
        const int hy = y0 + hj, hz = z0 + hk;
        const bool halo_on = has_halo && hy >= 0 && hy < ny && hz >= 0 && hz < nz;
        auto fill = [&](Real* dst) {
            for (int e = 0; e < P; e++) dst[e] = inf;
        };
        Real* const halo = T + ((hk + 2) * RY + hj + 2) * P;
        if (!row_on) fill(T + slot * P);
        if (has_halo && !halo_on) fill(halo);
        // What earlier visits wrote to the rows (bulk copies of other blocks) and read here is ordered
        // before these copies.
        asm volatile("fence.proxy.async;" ::: "memory");
        rows_expect(bar, (row_on ? P * 8u : 0u) + (halo_on ? P * 8u : 0u));
        if (row_on) row_in(smem_addr(T + slot * P), fd.T + rowi * pitch + x0, P * 8, bar);
        if (halo_on) row_in(smem_addr(halo), fd.T + (int64_t(hz) * ny + hy) * pitch + x0, P * 8, bar);
    }
    static_assert(4 * (BY + BZ) <= B::kThreads, "one halo row per thread");
    // The row's weights, fixed (seed or off-grid) and due nodes.
    const Real* __restrict__ srow = fd.s + rowi * nx + x0;
    const Real* wxp = static_cast<const Real*>(g.wx);
    const Real* wyp = static_cast<const Real*>(g.wy);
    const Real wx1 = ldg_r(&wxp[2 * rowi]), wx2 = ldg_r(&wxp[2 * rowi + 1]);
    const Real wy1 = ldg_r(&wyp[row_on ? 2 * gz : 0]), wy2 = ldg_r(&wyp[row_on ? 2 * gz + 1 : 1]);
    const Real wz1 = Real(g.wz1), wz2 = Real(g.wz2);
    const Real* zc = VARZ ? static_cast<const Real*>(g.zc) + kZCoef * (row_on ? gz : 0) : nullptr;
    uint32_t fixed = 0;
    {
        const bool in_range = tid >= fd.seed_tile_lo && tid <= fd.seed_tile_hi;
        int lo = 0, hi = in_range ? fd.seed_count : 0;
        while (lo < hi) {
            int mid = (lo + hi) >> 1;
            if (__ldg(&a.seed_tile[fd.seed_begin + mid]) < tid) lo = mid + 1;
            else hi = mid;
        }
        if (in_range && lo < fd.seed_count && __ldg(&a.seed_tile[fd.seed_begin + lo]) == tid)
            fixed = __ldg(&a.seed_mask[int64_t(fd.seed_begin + lo) * B::MW + k * BY + j]);
        if (!row_on) fixed = 0xffffffffu;
        else if (x0 + BX > nx) fixed |= ~((1u << (nx - x0)) - 1u);
    }
    // The due bits as bytes: four at a time (bits 0..3 of n become the bytes of n · 0x204081).
    const uint32_t due0 = __ldcg(&fd.dmask[int64_t(tid) * B::MW + k * BY + j]) & ~fixed;
    for (int q = t; q < B::kDueBytes / 4; q += B::kThreads) reinterpret_cast<uint32_t*>(due)[q] = 0u;
    __syncthreads();
    uint32_t* const row_due = reinterpret_cast<uint32_t*>(due + slot * DP + 4);
#pragma unroll
    for (int e = 0; e < BX / 4; e++) row_due[e] = (((due0 >> (4 * e)) & 15u) * 0x204081u) & 0x01010101u;
    if (t == 0) __stcg(&fd.dirty[tid], (uint8_t)0);
    const int off = (my ? BY - 1 - j : j) + (mz ? BZ - 1 - k : k);  // canonical j' + k'
    const uint32_t canon0 = mx ? __brev(due0) : due0;
    {
        const int first = __reduce_min_sync(0xffffffffu, canon0 ? off + __ffs(canon0) - 1 : B::NSTEPS);
        if (lane == 0) sh->first[warp] = first;
    }
    bool arrived = false;
    for (int q = 0; q < kMaxRowWaits && !arrived; q++) arrived = rows_arrived(smem_addr(&sh->arrived), parity);
    if (!__syncthreads_and(arrived)) {  // never seen: the copies did not come in about a second
        if (t == 0) {
            atomicCAS(&a.ctl->error, 0, TS_E_TIMEOUT);
            atomicExch(&a.ctl->abort, 1);
        }
        return 0;
    }

    const Real tol = a.tol, wake_rel = a.wake_rel;
    const bool causal = a.causal != 0;
    // The first plane that holds a due node: nothing can be woken before it.
    int p = B::NSTEPS;
#pragma unroll
    for (int w = 0; w < B::kThreads / 32; w++) p = min(p, sh->first[w]);
    // This warp's planes: outside them a step is only its barrier.
    const int wlo = __reduce_min_sync(0xffffffffu, off), whi = __reduce_max_sync(0xffffffffu, off) + BX - 1;
    bool big = false, mod = false;
    int evals = 0, woke = -4;  // woke: the last plane in which the thread woke a node
    // The thread's node of the plane and what lies at it move one node per plane.
    const int di = mx ? -1 : 1;
    int i = mx ? BX - 1 + off - p : p - off;  // off the row outside [0, BX)
    Real* c = T + slot * P + B::HX + i;
    uint8_t* d = due + slot * DP + 4 + i;
    // Slowness two planes ahead, where the row has a node then.
    const int xn = row_on ? min(BX, nx - x0) : 0;
    const Real* sp = srow + i;
    auto slow_at = [&](int q) -> Real { return unsigned(i + q * di) < unsigned(xn) ? ldg_r(sp + q * di) : Real(0); };
    const int skip = max(wlo - p, 0);  // to the warp's first plane
    Real s1 = slow_at(skip), s2 = slow_at(skip + 1);
    // A wake reaches the neighbours holding more than the new time (causal rule), or all.
    const Real none = minus_inf<Real>();
    for (; p < B::NSTEPS; p++) {
        const Real s0 = s1;
        if (p >= wlo && p <= whi) {
            s1 = s2;
            s2 = slow_at(2);
            if (unsigned(i) < unsigned(BX) && *(volatile uint8_t*)d && !((fixed >> i) & 1u)) {
                *d = 0;
                evals++;
                const Real cur = c[0];
                const Real xm = c[-1], xp = c[1], xm2 = c[-2], xp2 = c[2];
                const Real ym = c[-P], yp = c[P], ym2 = c[-2 * P], yp2 = c[2 * P];
                const Real zm = c[-L], zp = c[L], zm2 = c[-2 * L], zp2 = c[2 * L];
                const Real cand = Update<Real, VARZ>::eval(s0, xm, xp, xm2, xp2, ym, yp, ym2, yp2, zm, zp, zm2, zp2,
                                                           wx1, wx2, wy1, wy2, wz1, wz2, zc, second);
                if (cand < cur) {
                    c[0] = cand;
                    mod = true;
                    if (counts_as_change<Real>(cur, cand, tol)) big = true;
                    if (wakes<Real>(cur, cand, wake_rel)) {
                        const Real over = causal ? cand : none;
                        woke = p;
                        if (over < xm) d[-1] = 1;
                        if (over < xp) d[1] = 1;
                        if (over < xm2) d[-2] = 1;
                        if (over < xp2) d[2] = 1;
                        if (over < ym) d[-DP] = 1;
                        if (over < yp) d[DP] = 1;
                        if (over < ym2) d[-2 * DP] = 1;
                        if (over < yp2) d[2 * DP] = 1;
                        if (over < zm) d[-DL] = 1;
                        if (over < zp) d[DL] = 1;
                        if (over < zm2) d[-2 * DL] = 1;
                        if (over < zp2) d[2 * DL] = 1;
                    }
                }
            }
        }
        i += di;
        c += di;
        d += di;
        sp += di;
        // Every fourth plane the visit ends if nothing later can be due: no node that was due at its start
        // is left ahead, and the last two planes woke nothing.
        if ((p & 3) == 3) {
            const int ip = p + 1 - off;  // the thread's next node, canonical
            const bool ahead = ip <= 0 ? canon0 != 0u : ip < BX && (canon0 >> ip) != 0u;
            if (!__syncthreads_or(ahead || p - woke <= 1)) break;
        } else {
            __syncthreads();
        }
    }
    __syncthreads();

    // Hand the due nodes back; the changed rows; the neighbours' woken nodes.
    // (Four due bytes to bits: the sum of their shifts has them in its top four bits.)
    auto bits_of = [&](const uint32_t* w) {
        uint32_t v = 0;
#pragma unroll
        for (int e = 0; e < BX / 4; e++) v |= ((w[e] * 0x10204080u) >> 28) << (4 * e);
        return v;
    };
    const uint32_t left = bits_of(row_due) & ~fixed;
    __stcg(&fd.dmask[int64_t(tid) * B::MW + k * BY + j], left);
    if (__any_sync(0xffffffffu, left != 0u) && lane == 0) __stcg(&fd.dirty[tid], (uint8_t)1);
    if (mod) {  // the row's own thread alone wrote it
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        row_out(fd.T + rowi * pitch + B::HX + x0, smem_addr(T + slot * P + B::HX), BX * 8);
    }
    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
    auto wake_row = [&](int ntid, int r, uint32_t bits) {
        atomicOr(&fd.dmask[int64_t(ntid) * B::MW + r], bits);
        __stcg(&fd.dirty[ntid], (uint8_t)1);
    };
    for (int q = t; q < 4 * (BY + BZ); q += B::kThreads) {
        if (q < 4 * BZ) {  // y halo: rows −2, −1, BY, BY + 1 of each level
            const int e = q & 3, hk = q >> 2, hj = e < 2 ? e - 2 : BY + e - 2;
            const uint32_t bits = bits_of(reinterpret_cast<const uint32_t*>(due + ((hk + 2) * RY + hj + 2) * DP + 4));
            if (bits && y0 + hj >= 0 && y0 + hj < ny)
                wake_row(tid + (e < 2 ? -g.tx : g.tx), hk * BY + (e < 2 ? hj + BY : hj - BY), bits);
        } else {  // z halo
            const int h = q - 4 * BZ, e = h & 3, hj = h >> 2, hk = e < 2 ? e - 2 : BZ + e - 2;
            const uint32_t bits = bits_of(reinterpret_cast<const uint32_t*>(due + ((hk + 2) * RY + hj + 2) * DP + 4));
            if (bits && z0 + hk >= 0 && z0 + hk < nz)
                wake_row(tid + (e < 2 ? -1 : 1) * g.tx * g.ty, (e < 2 ? hk + BZ : hk - BZ) * BY + hj, bits);
        }
    }
    {  // x halo: x = −2, −1 before the row's nodes, BX, BX + 1 after them
        const uint8_t* d = due + slot * DP + 4;
        const uint32_t lo = (d[-1] ? 1u << 31 : 0u) | (d[-2] ? 1u << 30 : 0u);
        const uint32_t hi = (d[BX] ? 1u : 0u) | (d[BX + 1] ? 2u : 0u);
        if (lo && tx > 0) wake_row(tid - 1, k * BY + j, lo);
        if (hi && tx + 1 < g.tx) wake_row(tid + 1, k * BY + j, hi);
    }
    if (__any_sync(0xffffffffu, big) && lane == 0) __stcg(&fd.state->changed, 1);  // every writer writes 1
    asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    return evals;
}

// A tile per block: the blocks take due tiles from the queue, and a block that has finished one starts the
// tiles that waited for it last.
template <typename Real, int BX, int BY, int BZ, int MINB, bool VARZ_ANY>
__global__ void __launch_bounds__(BY * BZ, MINB) block_kernel(Args<Real> a) {
    using B = BlockTile<Real, BX, BY, BZ>;
    extern __shared__ __align__(16) unsigned char smem[];
    BlockShared* sh = reinterpret_cast<BlockShared*>(smem + B::kTimeBytes + B::kDueBytes);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned long long my_updates = 0, my_visits = 0;
    if (threadIdx.x == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(&sh->arrived)), "r"(B::kThreads) : "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    unsigned parity = 0;
    if (threadIdx.x == 0) atomicCAS(&a.ctl->t_start, 0ull, global_ns());
    // The scheduler's list lies where the due bytes are during a visit (never written by bulk copies).
    static_assert(B::kDueBytes >= 8 * kFlowList && B::kTimeBytes % 8 == 0, "room for the scheduler's list");
    unsigned long long* const list = reinterpret_cast<unsigned long long*>(smem + B::kTimeBytes);
    // Every running field starts its launch at the beginning of a round.
    for (int e = blockIdx.x; e < a.n_active; e += gridDim.x) {
        const int f = a.field_list[e];
        const FieldDesc<Real>& fd = a.fields[f];
        const GridDesc& g = fd.g;
        const int nt = g.tx * g.ty * g.tz;
        for (int q = threadIdx.x; q < nt; q += B::kThreads)
            __stcg(&fd.tokens[q], tokens_at_start(g, q % g.tx, q / g.tx % g.ty, q / (g.tx * g.ty)));
        if (threadIdx.x == 0) fd.state->launch_rounds = 0;
        __threadfence();
        __syncthreads();
        if (warp == 0) flow_run<Real, B::MW>(a, f, *(volatile const int*)&fd.state->phase, list, 0, lane);
        __syncthreads();
    }
    for (;;) {
        if (threadIdx.x == 0) sh->entry = queue_pop(a);
        __syncthreads();
        const unsigned long long item = sh->entry;
        if (item == 0ull) break;
        const TileItem it(item);
        const FieldDesc<Real>& fd = a.fields[it.field];
        if (VARZ_ANY && fd.g.varz) my_updates += visit_block<Real, BX, BY, BZ, true>(a, fd, it, smem, sh, parity);
        else my_updates += visit_block<Real, BX, BY, BZ, false>(a, fd, it, smem, sh, parity);
        my_visits += 1;
        parity ^= 1u;
        __syncthreads();
        if (warp == 0) {  // (the other warps wait for the next item)
            if (lane == 0) list[0] = TileItem::pack(it.tx, it.ty, it.tz, it.dir, it.phase, it.field);
            __syncwarp();
            flow_run<Real, B::MW>(a, it.field, it.phase, list, 1, lane);
        }
    }
    for (int o = 16; o > 0; o >>= 1) my_updates += __shfl_down_sync(0xffffffffu, my_updates, o);
    if (lane == 0) atomicAdd(&a.ctl->updates, my_updates);
    if (threadIdx.x == 0) atomicAdd(&a.ctl->visits, my_visits);
}

}  // namespace eik
}  // namespace ts
