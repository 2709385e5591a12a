// One launch of the tiled engine over a set of fields (an epoch): the job's descriptors laid out in one
// device arena, the new fields initialised and seeded, the cooperative persistent launch, the fields'
// states read back.
#include <algorithm>
#include <cstring>
#include <string>
#include <vector>

#include "eik_block.cuh"
#include "eik_engine.h"

namespace ts {
namespace eik {

namespace {

// A host image of device memory: aligned sub-allocations, uploaded in one copy.
struct Arena {
    std::vector<uint8_t> h;
    size_t add(size_t bytes, size_t align = 16) {
        size_t off = (h.size() + align - 1) / align * align;
        h.resize(off + std::max<size_t>(bytes, 1), 0);
        return off;
    }
    template <typename T>
    T* at(size_t off) { return reinterpret_cast<T*>(h.data() + off); }
};

// New fields of an epoch: +inf everywhere (pads included), every tile and node due, state zero.
template <typename Real>
__global__ void init_fields_kernel(const FieldDesc<Real>* __restrict__ fields, const int* __restrict__ init_list, int mw) {
    const FieldDesc<Real>& fd = fields[init_list[blockIdx.y]];
    const GridDesc& g = fd.g;
    int64_t n = int64_t(g.pitch) * g.ny * g.nz;
    const Real inf = real_inf<Real>();
    const int64_t t0 = blockIdx.x * int64_t(blockDim.x) + threadIdx.x, stride = int64_t(gridDim.x) * blockDim.x;
    for (int64_t q = t0; q < n; q += stride) fd.T[q] = inf;
    int64_t nt = int64_t(g.tx) * g.ty * g.tz;
    for (int64_t q = t0; q < (nt + 15) / 16 * 16; q += stride) fd.dirty[q] = q < nt ? 1 : 0;
    for (int64_t q = t0; q < nt * mw; q += stride) fd.dmask[q] = 0xffffffffu;  // every node due (EikonalOpenCl.cs:411)
    if (t0 == 0) *fd.state = FieldState{};
}

template <typename Real>
__global__ void seed_fields_kernel(const FieldDesc<Real>* __restrict__ fields, const int* __restrict__ field_of, const int32_t* __restrict__ node,
                                   const double* __restrict__ t, int count) {
    int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= count) return;
    const FieldDesc<Real>& fd = fields[field_of[q]];
    const GridDesc& g = fd.g;
    int n = node[q], i = n % g.nx, row = n / g.nx;
    fd.T[int64_t(row) * g.pitch + Layout<Real>::HX + i] = Real(t[q]);
}

// The epoch's field states, gathered for one copy to the host.
template <typename Real>
__global__ void gather_states_kernel(const FieldDesc<Real>* __restrict__ fields, int nf, FieldState* __restrict__ out) {
    int f = blockIdx.x * blockDim.x + threadIdx.x;
    if (f < nf) out[f] = *fields[f].state;
}

template <typename Real, int BY, int BZ, int MINB>
int launch_epoch(ts_ctx* ctx, const std::vector<const host::Grid*>& grids, const std::vector<const host::Metric*>& metrics,
                 const std::vector<EngineField*>& fl, double tol, double wake_rel, int max_rounds, ts_eik_stats* stats,
                 cudaStream_t s) {
    constexpr int BX = kTileX;
    using B = BlockTile<Real, BX, BY, BZ>;
    const int nf = int(fl.size());
    if (nf >= kMaxFields) return ctx->fail(TS_E_ARG, "too many fields in one launch");
    const int ng = int(grids.size());
    bool any_var = false;
    for (auto* g : grids) any_var |= g->variable;

    Arena A;
    // Grids.
    std::vector<size_t> o_wx(ng), o_wy(ng), o_zc(ng);
    std::vector<int> tx(ng), ty(ng), tz(ng);
    std::vector<GridDesc> descs(ng);
    for (int gi = 0; gi < ng; gi++) {
        const host::Grid& g = *grids[gi];
        const host::Metric& m = *metrics[gi];
        tx[gi] = (g.nx + BX - 1) / BX;
        ty[gi] = (g.ny + BY - 1) / BY;
        tz[gi] = (g.nz + BZ - 1) / BZ;
        if (tx[gi] > kMaxTilesX || ty[gi] > kMaxTilesYZ || tz[gi] > kMaxTilesYZ)
            return ctx->fail(TS_E_ARG, "grid too large for the tile table");
        o_wx[gi] = A.add(sizeof(Real) * m.wx.size());
        for (size_t q = 0; q < m.wx.size(); q++) A.at<Real>(o_wx[gi])[q] = Real(weight_of<Real>(m.wx[q], m.wx32[q]));
        o_wy[gi] = A.add(sizeof(Real) * m.wy.size());
        for (size_t q = 0; q < m.wy.size(); q++) A.at<Real>(o_wy[gi])[q] = Real(weight_of<Real>(m.wy[q], m.wy32[q]));
        o_zc[gi] = A.add(sizeof(Real) * std::max<size_t>(1, m.zc.size()));
        for (size_t q = 0; q < m.zc.size(); q++) A.at<Real>(o_zc[gi])[q] = Real(m.zc[q]);
    }
    // Seed tiles of each field (sorted by tile id) with their fixed-node masks; seed writes of the
    // fields this epoch initialises.
    std::vector<int> seed_begin(nf), seed_count(nf);
    std::vector<int> st_tile;
    std::vector<uint32_t> st_mask;
    std::vector<int> sc_field, init_list;
    std::vector<int32_t> sc_node;
    std::vector<double> sc_t;
    constexpr int kShape = BX | (BY << 8) | (BZ << 16);
    for (int f = 0; f < nf; f++) {
        EngineField& ef = *fl[f];
        const host::Grid& g = *grids[ef.grid];
        const int gi = ef.grid;
        if (!ef.initialized) {
            init_list.push_back(f);
            for (size_t q = 0; q < ef.seed_idx.size(); q++) {
                sc_field.push_back(f);
                sc_node.push_back(ef.seed_idx[q]);
                sc_t.push_back(ef.seed_t[q]);
            }
        }
        if (ef.seed_shape != kShape) {
            std::vector<std::pair<int, int>> tl;  // (tile, local)
            for (size_t q = 0; q < ef.seed_idx.size(); q++) {
                int node = ef.seed_idx[q];
                int i = node % g.nx, j = (node / g.nx) % g.ny, k = node / (g.nx * g.ny);
                int tid = ((k / BZ) * ty[gi] + j / BY) * tx[gi] + i / BX;
                int loc = ((k % BZ) * BY + j % BY) * BX + i % BX;
                tl.push_back({tid, loc});
            }
            std::sort(tl.begin(), tl.end());
            ef.seed_tiles.clear();
            ef.seed_masks.clear();
            for (size_t q = 0; q < tl.size(); q++) {
                if (q == 0 || tl[q].first != tl[q - 1].first) {
                    ef.seed_tiles.push_back(tl[q].first);
                    ef.seed_masks.resize(ef.seed_masks.size() + B::MW, 0u);
                }
                ef.seed_masks[(ef.seed_tiles.size() - 1) * B::MW + tl[q].second / 32] |= 1u << (tl[q].second % 32);
            }
            ef.seed_shape = kShape;
        }
        seed_begin[f] = int(st_tile.size());
        st_tile.insert(st_tile.end(), ef.seed_tiles.begin(), ef.seed_tiles.end());
        st_mask.insert(st_mask.end(), ef.seed_masks.begin(), ef.seed_masks.end());
        seed_count[f] = int(ef.seed_tiles.size());
    }
    size_t o_seed_tile = A.add(sizeof(int) * std::max<size_t>(1, st_tile.size()));
    std::copy(st_tile.begin(), st_tile.end(), A.at<int>(o_seed_tile));
    size_t o_seed_mask = A.add(sizeof(uint32_t) * std::max<size_t>(1, st_mask.size()));
    std::copy(st_mask.begin(), st_mask.end(), A.at<uint32_t>(o_seed_mask));
    size_t o_sc_field = A.add(sizeof(int) * sc_field.size());
    std::copy(sc_field.begin(), sc_field.end(), A.at<int>(o_sc_field));
    size_t o_sc_node = A.add(sizeof(int32_t) * sc_node.size());
    std::copy(sc_node.begin(), sc_node.end(), A.at<int32_t>(o_sc_node));
    size_t o_sc_t = A.add(sizeof(double) * sc_t.size(), 8);
    std::copy(sc_t.begin(), sc_t.end(), A.at<double>(o_sc_t));
    size_t o_init = A.add(sizeof(int) * init_list.size());
    std::copy(init_list.begin(), init_list.end(), A.at<int>(o_init));
    // The running fields.
    std::vector<int> field_list;
    for (int f = 0; f < nf; f++)
        if (fl[f]->status == 0) field_list.push_back(f);
    const int running = int(field_list.size());
    size_t o_field_list = A.add(sizeof(int) * std::max<size_t>(1, field_list.size()));
    std::copy(field_list.begin(), field_list.end(), A.at<int>(o_field_list));
    // The queue: room for every tile of every field (a tile is in it once at most, so that a producer never
    // waits for a consumer).
    size_t qcap = 1024, need = 0;
    for (int f : field_list) need += size_t(tx[fl[f]->grid]) * ty[fl[f]->grid] * tz[fl[f]->grid];
    while (qcap < need) qcap *= 2;
    // Fields, control, state copies.
    size_t o_fields = A.add(sizeof(FieldDesc<Real>) * nf);
    size_t o_ctl = A.add(sizeof(Control));
    size_t o_states = A.add(sizeof(FieldState) * nf);

    uint8_t* D = static_cast<uint8_t*>(ctx->buf("eng.arena", A.h.size()));
    if (!D) return TS_E_NOMEM;
    auto* q_slots = static_cast<unsigned long long*>(ctx->buf("eng.q_slots", 8 * qcap));
    if (!q_slots) return TS_E_NOMEM;
    auto* tokens = static_cast<unsigned*>(ctx->buf("eng.tokens", 4 * std::max<size_t>(1, need)));
    if (!tokens) return TS_E_NOMEM;
    for (int gi = 0; gi < ng; gi++) {
        GridDesc gd{};
        const host::Grid& g = *grids[gi];
        gd.nx = g.nx; gd.ny = g.ny; gd.nz = g.nz;
        gd.tx = tx[gi]; gd.ty = ty[gi]; gd.tz = tz[gi];
        gd.varz = g.variable ? 1 : 0;
        gd.wx = D + o_wx[gi];
        gd.wy = D + o_wy[gi];
        gd.zc = D + o_zc[gi];
        gd.wz1 = weight_of<Real>(metrics[gi]->wz1, metrics[gi]->wz1_32);
        gd.wz2 = weight_of<Real>(metrics[gi]->wz2, metrics[gi]->wz2_32);
        gd.pitch = Layout<Real>::pitch(tx[gi], BX);
        descs[gi] = gd;
    }
    for (int f = 0; f < nf; f++) {
        const EngineField& ef = *fl[f];
        FieldDesc<Real> fd{};
        fd.T = static_cast<Real*>(ef.T);
        fd.s = static_cast<const Real*>(ef.slowness);
        fd.dirty = ef.dirty;
        fd.dmask = ef.dmask;
        if (ef.status == 0) {
            fd.tokens = tokens;
            tokens += size_t(tx[ef.grid]) * ty[ef.grid] * tz[ef.grid];
        }
        fd.g = descs[ef.grid];
        fd.seed_begin = seed_begin[f];
        fd.seed_count = seed_count[f];
        fd.cap = ef.cap;
        fd.seed_tile_lo = seed_count[f] ? st_tile[seed_begin[f]] : 1;
        fd.seed_tile_hi = seed_count[f] ? st_tile[seed_begin[f] + seed_count[f] - 1] : 0;
        fd.state = static_cast<FieldState*>(ef.state);
        A.at<FieldDesc<Real>>(o_fields)[f] = fd;
    }
    A.at<Control>(o_ctl)->running = running;

    // The work of the epoch, enqueued on stream s: arena upload (from a pinned image), new fields'
    // initialisation and seeds, the engine launch, and the control block and field states back to
    // pinned host memory. Recorded directly, or captured once into a CUDA graph and replayed while
    // the same job (same arena bytes, same buffers) is solved again.
    uint8_t* image = static_cast<uint8_t*>(ctx->host_buf("eng.arena.image", A.h.size()));
    Control* ctl_h = static_cast<Control*>(ctx->host_buf("eng.ctl", sizeof(Control)));
    FieldState* st_h = static_cast<FieldState*>(ctx->host_buf("eng.states", sizeof(FieldState) * std::max(1, nf)));
    if (!image || !ctl_h || !st_h) return TS_E_NOMEM;
    std::memcpy(image, A.h.data(), A.h.size());
    *ctl_h = Control{};

    Args<Real> args;
    std::memset(static_cast<void*>(&args), 0, sizeof args);  // its bytes are part of a captured job's signature
    args.fields = reinterpret_cast<const FieldDesc<Real>*>(D + o_fields);
    args.seed_tile = reinterpret_cast<const int*>(D + o_seed_tile);
    args.seed_mask = reinterpret_cast<const uint32_t*>(D + o_seed_mask);
    args.ctl = reinterpret_cast<Control*>(D + o_ctl);
    args.cancel = ctx->cancel_dev;
    args.field_list = reinterpret_cast<const int*>(D + o_field_list);
    args.n_active = running;
    args.max_rounds_per_launch = max_rounds;
    args.epoch_budget_ns = (ctx->scheduler == 1 && max_rounds > 0) ? (long long)(ctx->epoch_budget_ms * 1e6) : 0;
    args.barrier_timeout_ns = 5000000000LL;
    args.q_slots = q_slots;
    args.q_mask = qcap - 1;
    for (args.q_bits = 0; (size_t(1) << args.q_bits) < qcap;) args.q_bits++;
    args.tol = Real(tol);
    args.wake_rel = Real(wake_rel);
    args.causal = wake_rel > 0 ? 1 : 0;  // fast mode: threshold and causal wakes together
    const int smem = B::kBytes;
    void* kfn = any_var ? (void*)block_kernel<Real, BX, BY, BZ, MINB, true> : (void*)block_kernel<Real, BX, BY, BZ, MINB, false>;
    TS_CUDA_TRY(ctx, cudaFuncSetAttribute(kfn, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    int per_sm = 0;
    TS_CUDA_TRY(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kfn, B::kThreads, smem));
    if (per_sm < 1) return ctx->fail(TS_E_CUDA, "engine kernel does not fit on an SM");
    // No more blocks than tiles.
    const int blocks = int(std::min<size_t>(size_t(per_sm) * ctx->sm_count, std::max<size_t>(1, need)));
    void* params[] = {&args};
    int64_t maxn = 0;
    for (int f : init_list) {
        const host::Grid& g = *grids[fl[f]->grid];
        maxn = std::max(maxn, int64_t(Layout<Real>::pitch(tx[fl[f]->grid], BX)) * g.ny * g.nz);
    }
    cudaEvent_t k0 = nullptr, k1 = nullptr;
    auto enqueue = [&](bool timed) -> cudaError_t {
        cudaError_t e = cudaMemcpyAsync(D, image, A.h.size(), cudaMemcpyHostToDevice, s);
        if (e != cudaSuccess) return e;
        for (size_t c0 = 0; c0 < init_list.size(); c0 += 65535) {
            unsigned cnt = unsigned(std::min<size_t>(65535, init_list.size() - c0));
            dim3 grid(unsigned(std::min<int64_t>((maxn + 255) / 256, 512)), cnt);
            init_fields_kernel<Real><<<grid, 256, 0, s>>>(reinterpret_cast<const FieldDesc<Real>*>(D + o_fields),
                                                          reinterpret_cast<const int*>(D + o_init) + c0, B::MW);
        }
        int cnt = int(sc_node.size());
        if (cnt > 0)
            seed_fields_kernel<Real><<<(cnt + 255) / 256, 256, 0, s>>>(
                reinterpret_cast<const FieldDesc<Real>*>(D + o_fields), reinterpret_cast<const int*>(D + o_sc_field), reinterpret_cast<const int32_t*>(D + o_sc_node),
                reinterpret_cast<const double*>(D + o_sc_t), cnt);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
        if (running > 0 && (e = cudaMemsetAsync(q_slots, 0, 8 * qcap, s)) != cudaSuccess) return e;
        if (running > 0) {
            if (timed) cudaEventRecord(k0, s);
            e = cudaLaunchCooperativeKernel(kfn, dim3(blocks), dim3(B::kThreads), params, smem, s);
            if (timed) cudaEventRecord(k1, s);
            if (e != cudaSuccess) return e;
        }
        gather_states_kernel<Real><<<(nf + 127) / 128, 128, 0, s>>>(reinterpret_cast<const FieldDesc<Real>*>(D + o_fields),
                                                                    nf, reinterpret_cast<FieldState*>(D + o_states));
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
        if ((e = cudaMemcpyAsync(ctl_h, D + o_ctl, sizeof(Control), cudaMemcpyDeviceToHost, s)) != cudaSuccess) return e;
        return cudaMemcpyAsync(st_h, D + o_states, sizeof(FieldState) * nf, cudaMemcpyDeviceToHost, s);
    };
    bool graphed = false;
    if (ctx->use_graph && max_rounds <= 0) {
        // The job's signature: its arena bytes, the buffers the work touches and what the captured launches
        // were given by value (the kernel's arguments: the settle tolerance and the mode's wake rule among them).
        unsigned long long sig = 1469598103934665603ULL;
        auto mix = [&](const void* p, size_t n) {
            const uint8_t* b = static_cast<const uint8_t*>(p);
            for (size_t q = 0; q < n; q++) sig = (sig ^ b[q]) * 1099511628211ULL;
        };
        mix(A.h.data(), A.h.size());
        const uintptr_t ptrs[] = {uintptr_t(D), uintptr_t(q_slots), uintptr_t(image), uintptr_t(ctl_h), uintptr_t(st_h), uintptr_t(kfn)};
        mix(ptrs, sizeof ptrs);
        const uint64_t sizes[] = {A.h.size(), o_init, init_list.size(), sc_node.size(), o_sc_node, o_states, size_t(nf), size_t(maxn),
                                  qcap, size_t(running), size_t(blocks), size_t(smem)};
        mix(sizes, sizeof sizes);
        mix(&args, sizeof args);
        if (ctx->graph_exec && ctx->graph_sig == sig) {
            TS_CUDA_TRY(ctx, cudaGraphLaunch(ctx->graph_exec, s));
            ctx->graph_replays++;
            graphed = true;
        } else {
            ctx->drop_graph();
            cudaGraph_t graph = nullptr;
            cudaError_t e = cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal);
            if (e == cudaSuccess) {
                cudaError_t we = enqueue(false);
                e = cudaStreamEndCapture(s, &graph);
                if (we != cudaSuccess) e = we;
            }
            if (e == cudaSuccess && graph) e = cudaGraphInstantiate(&ctx->graph_exec, graph, 0);
            if (graph) cudaGraphDestroy(graph);
            if (e == cudaSuccess && ctx->graph_exec) {
                ctx->graph_sig = sig;
                TS_CUDA_TRY(ctx, cudaGraphLaunch(ctx->graph_exec, s));
                graphed = true;
            } else {
                cudaGetLastError();  // capture unsupported here: run the work directly
                ctx->drop_graph();
            }
        }
    }
    if (!graphed) {
        cudaEventCreate(&k0);
        cudaEventCreate(&k1);
        cudaError_t e = enqueue(true);
        if (e != cudaSuccess) {
            cudaEventDestroy(k0);
            cudaEventDestroy(k1);
            TS_CUDA_TRY(ctx, e);
        }
    }
    TS_CUDA_TRY(ctx, cudaStreamSynchronize(s));
    for (int f : init_list) fl[f]->initialized = true;
    const Control ctl = *ctl_h;
    float kms = 0;
    if (!graphed && running > 0) cudaEventElapsedTime(&kms, k0, k1);
    if (k0) cudaEventDestroy(k0);
    if (k1) cudaEventDestroy(k1);
    if (stats) {
        stats->kernel_ms += kms;
        stats->node_updates += int64_t(ctl.updates);
        stats->tile_visits += int64_t(ctl.visits);
        stats->launches += running > 0 ? 1 : 0;
    }
    std::vector<FieldState> st(st_h, st_h + nf);
    for (int f = 0; f < nf; f++) {
        fl[f]->status = st[f].status;
        fl[f]->rounds[0] = st[f].rounds0;
        fl[f]->rounds[1] = st[f].rounds1;
    }
    if (ctl.error == TS_E_CANCELLED) return ctx->fail(TS_E_CANCELLED, "cancelled");
    if (ctl.error) return ctx->fail(ctl.error, "engine: a device-side wait ran out");
    return TS_OK;
}

}  // namespace

template <typename Real>
int engine_epoch(ts_ctx* ctx, const std::vector<const host::Grid*>& grids,
                 const std::vector<const host::Metric*>& metrics, const std::vector<EngineField*>& fields,
                 double tol, double wake_rel, int max_rounds, ts_eik_stats* stats, cudaStream_t s) {
    if (fields.empty()) return TS_OK;
    // Three blocks per SM, as their shared memory (77 KB each) and their registers (156 to 164 a thread in FP64)
    // allow.
    return launch_epoch<Real, kTileY, kTileZ, 3>(ctx, grids, metrics, fields, tol, wake_rel, max_rounds, stats, s);
}

template int engine_epoch<Pair>(ts_ctx*, const std::vector<const host::Grid*>&, const std::vector<const host::Metric*>&,
                                 const std::vector<EngineField*>&, double, double, int, ts_eik_stats*, cudaStream_t);
template int engine_epoch<double>(ts_ctx*, const std::vector<const host::Grid*>&, const std::vector<const host::Metric*>&,
                                  const std::vector<EngineField*>&, double, double, int, ts_eik_stats*, cudaStream_t);

}  // namespace eik
}  // namespace ts
