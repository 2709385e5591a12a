// How the engine's fields advance: one launch over many fields and grids, no grid-wide barrier.
#pragma once

#include "eik_kernels.cuh"

namespace ts {
namespace eik {

// ---- flow scheduler: no grid-wide barrier; each field advances on its own ----------------------
//
// A field's sweep needs only that a tile diagonal q is done before diagonal q+1 of the same field
// starts (the order argument of the engine); fields are independent. So each field keeps its own
// position (ordering, diagonal) and count of outstanding tiles; its due tiles go into one global
// queue that every block of the launch takes from. The warp that finishes a field's last tile of a
// diagonal advances that field: it finds the next diagonal with due tiles (across sweeps and round
// ends, which it evaluates for that field alone) and queues them. A launch ends when every field
// has settled, been refused at the cap, been cancelled, or run its rounds for this launch. Waits
// for a queue slot are bounded (globaltimer); a wait that runs out raises the abort flag and the
// launch ends with TS_E_TIMEOUT.

// Ends a round of field f (SphericalEikonal.cs:297-323; EikonalOpenCl.cs:241-269). Whole warp.
// Returns true when the field stops in this launch.
template <typename Real, int MW>
TS_DEVINL bool flow_round_end(const Args<Real>& a, int f, int lane, int& phase) {
    const FieldDesc<Real>& fd = a.fields[f];
    volatile FieldState* st = fd.state;
    bool stop = false, fill = false;
    if (lane == 0) {
        const int cap = fd.cap;
        if (!st->changed) {
            if (st->phase == 0) {
                st->rounds0 = st->round + 1;
                st->phase = 1;
                st->round = 0;
                fill = true;  // phase 1 starts with every node due (EikonalOpenCl.cs:235-239)
            } else {
                st->rounds1 = st->round + 1;
                st->status = kSettled;
                stop = true;
            }
        } else {
            st->round = st->round + 1;
            if (st->round >= cap) {
                if (st->phase == 0) st->rounds0 = st->round;
                else st->rounds1 = st->round;
                st->status = kUnsettled;
                stop = true;
            }
        }
        st->changed = 0;
        st->launch_rounds = st->launch_rounds + 1;
        if (!stop && a.max_rounds_per_launch > 0 && st->launch_rounds >= a.max_rounds_per_launch) stop = true;
        if (!stop && a.epoch_budget_ns > 0 &&
            (long long)(global_ns() - *(volatile unsigned long long*)&a.ctl->t_start) > a.epoch_budget_ns)
            stop = true;
        if (!stop && a.cancel && *a.cancel) {
            atomicCAS(&a.ctl->error, 0, TS_E_CANCELLED);
            stop = true;
        }
    }
    stop = __shfl_sync(0xffffffffu, stop, 0);
    fill = __shfl_sync(0xffffffffu, fill, 0);
    if (fill) phase = 1;
    if (fill) {
        const GridDesc& g = fd.g;
        const int64_t nt = int64_t(g.tx) * g.ty * g.tz;
        for (int64_t q = lane; q < nt; q += 32) __stcg(&fd.dirty[q], (uint8_t)1);
        for (int64_t q = lane; q < nt * MW; q += 32) __stcg(&fd.dmask[q], 0xffffffffu);
    }
    return stop;
}

// A tile in the queue: the tile's coordinates, the sweep ordering and phase it is due in, its field, and
// the lap (1..63) of its ticket, so that a visit starts from the word alone.
struct TileItem {
    int tx, ty, tz, dir, phase, field;
    TS_DEVINL static unsigned long long pack(int tx, int ty, int tz, int dir, int phase, int field) {
        return (unsigned long long)(unsigned(tx) | (unsigned(ty) << 10) | (unsigned(tz) << 20)) |
               ((unsigned long long)(unsigned(dir) | (unsigned(phase) << 3) | (unsigned(field) << 4)) << 30);
    }
    TS_DEVINL explicit TileItem(unsigned long long w)
        : tx(int(w & 1023u)), ty(int((w >> 10) & 1023u)), tz(int((w >> 20) & 1023u)), dir(int((w >> 30) & 7u)),
          phase(int((w >> 33) & 1u)), field(int((w >> 34) & 0xffffffu)) {}
};
constexpr int kMaxFields = 1 << 24, kLapShift = 58;
template <typename Real>
TS_DEVINL unsigned long long lap_of(const Args<Real>& a, unsigned long long ticket) {
    return (1ull + (ticket >> a.q_bits) % 63ull) << kLapShift;
}

// Moves field f to its next diagonal with due tiles, from diagonal q of ordering dir on, and queues those
// tiles; or stops the field. Whole warp.
template <typename Real, int MW>
TS_DEVINL void flow_advance(const Args<Real>& a, int f, int dir, int q, int phase, int lane) {
    const FieldDesc<Real>& fd = a.fields[f];
    const GridDesc& g = fd.g;
    volatile FieldState* st = fd.state;
    for (;;) {
        if (q >= g.ndiag) {
            q = 0;
            if (++dir == 8) {
                dir = 0;
                __threadfence();
                const bool stopped = flow_round_end<Real, MW>(a, f, lane, phase);
                __threadfence();
                __syncwarp();
                if (stopped) {
                    if (lane == 0) {
                        st->pending = 0;
                        if (atomicSub(&a.ctl->running, 1) == 1) atomicExch(&a.ctl->done, 1);
                    }
                    __syncwarp();
                    return;
                }
            }
        }
        auto tile = [&](int e, int& tx, int& ty, int& tz) {
            const uint32_t pk = __ldg(&g.diag_tiles[e]);
            const int ca = pk & 1023, cb = (pk >> 10) & 1023, cc = pk >> 20;
            tx = (dir & 1) ? g.tx - 1 - ca : ca;
            ty = (dir & 2) ? g.ty - 1 - cb : cb;
            tz = (dir & 4) ? g.tz - 1 - cc : cc;
        };
        // Due tiles of diagonal q under ordering dir; none of them is visited before they are queued.
        const int d0 = __ldg(&g.diag_off[q]), cnt = __ldg(&g.diag_off[q + 1]) - d0;
        int due_total = 0;
        unsigned kept = 0;  // lane c: the due tiles of the c-th 32 of the diagonal (1,024 tiles in all)
        for (int b = 0; b < cnt; b += 32) {
            bool due = false;
            if (b + lane < cnt) {
                int tx, ty, tz;
                tile(d0 + b + lane, tx, ty, tz);
                due = __ldcg(&fd.dirty[(tz * g.ty + ty) * g.tx + tx]) != 0;
            }
            const unsigned m = __ballot_sync(0xffffffffu, due);
            if (lane == (b >> 5)) kept = m;
            due_total += __popc(m);
        }
        if (due_total == 0) {
            q++;
            continue;
        }
        // The count before the tiles: a consumer may finish one at once.
        if (lane == 0) st->pending = due_total;
        __syncwarp();
        __threadfence();
        unsigned long long base = 0;
        if (lane == 0) base = atomicAdd(&a.ctl->q_tail, (unsigned long long)due_total);
        base = __shfl_sync(0xffffffffu, base, 0);
        int written = 0;
        for (int b = 0; b < cnt; b += 32) {
            const unsigned have = __shfl_sync(0xffffffffu, kept, (b >> 5) & 31);
            bool due = b < 1024 && ((have >> lane) & 1u);
            unsigned long long item = 0;
            if (due || (b >= 1024 && b + lane < cnt)) {
                int tx, ty, tz;
                tile(d0 + b + lane, tx, ty, tz);
                if (b >= 1024) due = __ldcg(&fd.dirty[(tz * g.ty + ty) * g.tx + tx]) != 0;
                item = TileItem::pack(tx, ty, tz, dir, phase, f);
            }
            const unsigned m = __ballot_sync(0xffffffffu, due);
            if (due) {
                const unsigned long long ticket = base + written + __popc(m & ((1u << lane) - 1u));
                unsigned long long* const slot = &a.q_slots[ticket & a.q_mask];
                const unsigned long long t0 = global_ns();
                while (atomicCAS(slot, 0ull, item | lap_of(a, ticket)) != 0ull) {  // its last tile not taken yet
                    if (*(volatile int*)&a.ctl->abort || (long long)(global_ns() - t0) > a.barrier_timeout_ns) {
                        atomicCAS(&a.ctl->error, 0, TS_E_TIMEOUT);
                        atomicExch(&a.ctl->abort, 1);
                        break;
                    }
                    __nanosleep(64);
                }
            }
            written += __popc(m);
        }
        __syncwarp();
        return;
    }
}

}  // namespace eik
}  // namespace ts
