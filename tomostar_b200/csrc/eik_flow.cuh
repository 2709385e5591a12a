// How the engine's fields advance: one launch over many fields and grids, no grid-wide barrier.
#pragma once

#include "eik_kernels.cuh"

namespace ts {
namespace eik {

// ---- flow scheduler: no grid-wide barrier; each tile starts when its neighbours allow -----------
//
// A tile's sweep s reads the face neighbours before it along the sweep as that sweep left them and those
// after it as the sweep before did, and wakes nodes of all of them; so it may start when the former have
// finished sweep s, the latter sweep s − 1, and it itself sweep s − 1. Nothing else orders tiles: the
// tiles of a field run as a wave, and the next sweep's wave starts behind it as soon as its own first
// tiles are free (one axis or two keep their direction from one ordering to most of the next). Only a
// round's end waits for the whole field.
//
// Each tile counts what it waits for in tokens, a half word for even and one for odd sweeps: one from
// itself and one from each neighbour per sweep (a neighbour before it gives its token when it finishes
// the sweep, one after it when it finishes the sweep before). Whoever gives the last one starts the tile:
// with due nodes it goes into one global queue that every block of the launch takes from, without it is
// finished at once and gives its own tokens. Tokens for a sweep two later cannot come before the tile has
// finished this one, so two halves are enough. After a round the counts are those of its start.
//
// By diagonals (each started when the last tile of the one before was done) the blocks waited for the slowest
// tile of each and in the short ones at a sweep's ends: 56 % of their time went into visits with 50 fields of
// 121×121×61. Kernel time by diagonals and by tokens, in turn on one GPU: those 56.4 -> 43.5 ms, 16 uneven grids
// in FP32 57.9 -> 37.9, 24 of 401×401×121, which keep every block busy either way, 696 -> 717: the fields now
// advance evenly, and their rounds' ends coincide. (With a tile twice as deep, which has gone: 25 fields of
// 81×81×41 24.1 -> 17.8, 10 of 161×161×81 114 -> 97.)
// What did not help there: handing a started tile to the visit that started it, a warp of its own for the
// tokens that also takes the next tile during a visit, taking it by another warp while the tokens are given,
// and diagonals in the rounds that begin with few due tiles.
//
// A launch ends when every field has settled, been refused at the cap, been cancelled, or run its rounds
// for this launch. Waits for a queue slot are bounded (globaltimer); a wait that runs out raises the
// abort flag and the launch ends with TS_E_TIMEOUT.

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

// What a warp wrote or saw before is ordered before what it does after, for the whole GPU (lighter than
// the sequentially consistent __threadfence()).
TS_DEVINL void fence_gpu() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }

// A tile in the queue: the tile's coordinates (11, 10 and 10 bits), the sweep ordering and phase it is due in, its
// field, and the lap (1..31) of its ticket, so that a visit starts from the word alone.
struct TileItem {
    int tx, ty, tz, dir, phase, field;
    TS_DEVINL static unsigned long long pack(int tx, int ty, int tz, int dir, int phase, int field) {
        return (unsigned long long)(unsigned(tx) | (unsigned(ty) << 11) | (unsigned(tz) << 21)) |
               ((unsigned long long)(unsigned(dir) | (unsigned(phase) << 3) | (unsigned(field) << 4)) << kDirShift);
    }
    TS_DEVINL explicit TileItem(unsigned long long w)
        : tx(int(w & 2047u)), ty(int((w >> 11) & 1023u)), tz(int((w >> 21) & 1023u)), dir(int((w >> kDirShift) & 7u)),
          phase(int((w >> (kDirShift + 3)) & 1u)), field(int((w >> (kDirShift + 4)) & 0xffffffu)) {}
    static constexpr int kDirShift = 31;
    TS_DEVINL static int shift(int axis) { return axis == 0 ? 0 : 10 * axis + 1; }
};
constexpr int kMaxTilesX = 2048, kMaxTilesYZ = 1024, kMaxFields = 1 << 24, kLapShift = 59;
template <typename Real>
TS_DEVINL unsigned long long lap_of(const Args<Real>& a, unsigned long long ticket) {
    return (unsigned long long)(1u + unsigned(ticket >> a.q_bits) % 31u) << kLapShift;
}

// What a tile waits for: itself and its neighbours.
TS_DEVINL unsigned tokens_needed(int gx, int gy, int gz, int tx, int ty, int tz) {
    return 1u + unsigned(tx > 0) + unsigned(tx + 1 < gx) + unsigned(ty > 0) + unsigned(ty + 1 < gy) + unsigned(tz > 0) +
           unsigned(tz + 1 < gz);
}
// Tokens a tile holds before a round's first sweep: its own and those of the neighbours after it.
TS_DEVINL unsigned tokens_at_start(const GridDesc& g, int tx, int ty, int tz) {
    return 1u + unsigned(tx + 1 < g.tx) + unsigned(ty + 1 < g.ty) + unsigned(tz + 1 < g.tz);
}

// A tile into the slot of its ticket. The queue has a slot for every tile, so that the slot is free.
template <typename Real>
TS_DEVINL void queue_put(const Args<Real>& a, unsigned long long ticket, unsigned long long word) {
    unsigned long long* const slot = &a.q_slots[ticket & a.q_mask];
    if (atomicCAS(slot, 0ull, word | lap_of(a, ticket)) == 0ull) return;
    const unsigned long long t0 = global_ns();
    while (atomicCAS(slot, 0ull, word | lap_of(a, ticket)) != 0ull) {  // its last tile not taken yet
        if (*(volatile int*)&a.ctl->abort || (long long)(global_ns() - t0) > a.barrier_timeout_ns) {
            atomicCAS(&a.ctl->error, 0, TS_E_TIMEOUT);
            atomicExch(&a.ctl->abort, 1);
            return;
        }
        __nanosleep(64);
    }
}

// The next tile of the queue, its slot freed; waits for one. 0: the launch has ended or a wait ran out. One lane.
template <typename Real>
TS_DEVINL unsigned long long queue_pop(const Args<Real>& a) {
    const unsigned long long ticket = atomicAdd(&a.ctl->q_head, 1ull);
    volatile unsigned long long* const slot = &a.q_slots[ticket & a.q_mask];
    const unsigned long long lap = lap_of(a, ticket) >> kLapShift;
    // The limit counts from the last tiles any block queued: a long wait while others work is not a failure.
    unsigned long long t0 = global_ns(), seen = *(volatile unsigned long long*)&a.ctl->q_tail;
    for (unsigned polls = 1;; polls++) {
        const unsigned long long item = *slot;
        if (item >> kLapShift == lap) {
            *slot = 0ull;
            __threadfence();
            return item;
        }
        if (*(volatile int*)&a.ctl->done || *(volatile int*)&a.ctl->abort) return 0;
        if ((polls & 15u) == 0) {
            const unsigned long long now = *(volatile unsigned long long*)&a.ctl->q_tail;
            if (now != seen) {
                seen = now;
                t0 = global_ns();
            }
            if ((long long)(global_ns() - t0) > a.barrier_timeout_ns) {
                atomicCAS(&a.ctl->error, 0, TS_E_TIMEOUT);
                atomicExch(&a.ctl->abort, 1);
                return 0;
            }
        }
        __nanosleep(polls < 8 ? 32 : 128);
    }
}

// The field that a warp moves on, and where a lane stands in it: eight lanes per finished tile, for its six
// neighbours (axis, up) and itself (6).
struct FlowField {
    int gx, gy, gz;
    unsigned* tokens;
    const uint8_t* dirty;
    int lane, sub, axis, up;
};
constexpr int kFlowList = 1024;

// Gives the tokens of up to four finished tiles, the last of list[0..count); queues the due tiles that they
// start and appends those without due nodes to the list, as finished. ended += tiles that finished the
// round. False when the launch has been given up. Whole warp. A step is the latency of an atomic, a fence, a
// load and a queue slot, some 3 µs, whatever it carries, and most carry one tile (steps of sixteen tiles cost
// more instructions than they saved steps: 24 fields of 401×401×121 735 ms for 717).
template <typename Real>
TS_DEVINL bool flow_step(const Args<Real>& a, const FlowField& w, unsigned long long* list, int& count, int& ended) {
    const int n = min(count, 4), q = w.lane >> 3;
    count -= n;
    unsigned long long word = 0;
    unsigned add = 0, need = 0;
    int at = 0, s = 0;
    const bool self = w.sub == 6;
    if (q < n && w.sub < 7) {
        word = list[count + q];
        TileItem z(word);
        s = z.dir;
        const int even = 16 * (s & 1), odd = 16 - even;
        if (!self) {
            const int d = w.up ? 1 : -1;
            if (w.axis == 0) z.tx += d;
            else if (w.axis == 1) z.ty += d;
            else z.tz += d;
            const bool on = unsigned(z.tx) < unsigned(w.gx) && unsigned(z.ty) < unsigned(w.gy) && unsigned(z.tz) < unsigned(w.gz);
            // After the tile in sweep s: its token for s. Before it in s + 1: for s + 1.
            if (on && w.up != ((s >> w.axis) & 1)) add += 1u << even;
            if (on && w.up == (((s + 1) >> w.axis) & 1)) add += 1u << odd;
            word += (unsigned long long)(long long)d << TileItem::shift(w.axis);
        }
        at = (z.tz * w.gy + z.ty) * w.gx + z.tx;
        need = tokens_needed(w.gx, w.gy, w.gz, z.tx, z.ty, z.tz);
        if (self) {
            add = (1u << odd) - (need << even);
            ended += s == 7;
        }
    }
    const unsigned got = add ? atomicAdd(&w.tokens[at], add) + add : 0u;
    // (a lane without a neighbour looks whether the launch has been given up)
    if (__any_sync(0xffffffffu, w.sub == 7 && *(volatile int*)&a.ctl->abort)) return false;
    const int even = 16 * (s & 1), odd = 16 - even;
    const bool now = !self && (add >> even & 0xffffu) && (got >> even & 0xffffu) == need;
    const bool next = add && (self || (add >> odd & 0xffffu)) && (got >> odd & 0xffffu) == need && s < 7;
    const bool ready = now || next;
    if (next) word += 1ull << TileItem::kDirShift;
    if (!__any_sync(0xffffffffu, ready)) return true;
    fence_gpu();
    bool due = ready && __ldcg(&w.dirty[at]) != 0;
    // Tiles without due nodes to the list (the queue when it is full), the others to the queue.
    const unsigned before = (1u << w.lane) - 1u;
    const unsigned m = __ballot_sync(0xffffffffu, ready && !due);
    if (ready && !due) {
        const int at_q = count + __popc(m & before);
        if (at_q < kFlowList) list[at_q] = word;
        else due = true;
    }
    count = min(count + __popc(m), kFlowList);
    const unsigned to_queue = __ballot_sync(0xffffffffu, due);
    if (to_queue) {
        unsigned long long ticket = 0;
        if (w.lane == 0) ticket = atomicAdd(&a.ctl->q_tail, (unsigned long long)__popc(to_queue));
        ticket = __shfl_sync(0xffffffffu, ticket, 0);
        if (due) queue_put(a, ticket + __popc(to_queue & before), word);
    }
    __syncwarp();
    return true;
}

// Goes on with field f after the tiles in list[0..count) (queue words without lap: the tile and the sweep it
// finished; count 0: with a round): gives their tokens and those of the tiles without due nodes that start
// and finish at once, queues the due tiles that start, and ends rounds. `list` is shared memory with room
// for kFlowList words. Whole warp. (Not inlined: the visit keeps its registers.)
template <typename Real, int MW>
__device__ __noinline__ void flow_run(const Args<Real>& a, int f, int phase, unsigned long long* list, int count, int lane) {
    const FieldDesc<Real>& fd = a.fields[f];
    const int sub = lane & 7;
    // (in registers: a fence drops the L1 lines)
    const FlowField w{fd.g.tx, fd.g.ty, fd.g.tz, fd.tokens, fd.dirty, lane, sub, sub >> 1, sub & 1};
    const int nt = w.gx * w.gy * w.gz;
    FieldState* const st = fd.state;
    fence_gpu();  // what the block wrote comes before the tokens (later steps: the fence of the one before)
    bool begins = count == 0;
    for (;;) {
        bool idle = false;
        if (begins) {
            begins = false;
            // Nothing due anywhere: the round ends as it begins (a byte per tile, sixteen to a load; field
            // buffers are padded to 256 bytes, and the bytes after the last tile are zero).
            uint32_t some = 0;
            for (int q = 16 * lane; q < nt; q += 512) {
                const uint4 v = __ldcg(reinterpret_cast<const uint4*>(w.dirty + q));
                some |= v.x | v.y | v.z | v.w;
            }
            idle = !__any_sync(0xffffffffu, some != 0u);
            if (!idle) {
                if (lane == 0) *(volatile int*)&st->pending = nt;
                __syncwarp();
                fence_gpu();
                const unsigned long long word = TileItem::pack(0, 0, 0, 0, phase, f);
                if (__ldcg(&w.dirty[0])) {
                    if (lane == 0) queue_put(a, atomicAdd(&a.ctl->q_tail, 1ull), word);
                    __syncwarp();
                    return;
                }
                if (lane == 0) list[0] = word;
                count = 1;
                __syncwarp();
            }
        }
        int ended = 0;
        while (count > 0)
            if (!flow_step(a, w, list, count, ended)) return;
        // The round's end, once every tile has finished its last sweep.
        if (!idle) {
            ended = __reduce_add_sync(0xffffffffu, ended);
            if (!ended) return;
            int left = 1;
            if (lane == 0) {
                fence_gpu();
                left = atomicSub(&st->pending, ended) - ended;
            }
            if (__shfl_sync(0xffffffffu, left, 0) != 0) return;
        }
        fence_gpu();
        const bool stopped = flow_round_end<Real, MW>(a, f, lane, phase);
        fence_gpu();
        __syncwarp();
        if (stopped) {
            if (lane == 0 && atomicSub(&a.ctl->running, 1) == 1) atomicExch(&a.ctl->done, 1);
            __syncwarp();
            return;
        }
        begins = true;
    }
}

}  // namespace eik
}  // namespace ts
