// The tiled engine's host side: a job's buffers, its tile shape, its fields' way back to the host.
#include <algorithm>
#include <cstring>
#include <string>
#include <type_traits>
#include <vector>

#include "eik_engine.h"
#include "eik_kernels.cuh"
#include "eik_resident.h"
#include "host_copy.h"

namespace ts {
namespace eik {

// The tile shape compiled into the library; and the ids that callers may give: its own, or one of earlier
// libraries' shapes, for which it stands in. (A deeper tile of 32×16×16 nodes, one block per SM, crosses a grid
// in fewer and longer visits. Since tiles start as their neighbours allow it is behind everywhere, kernel time
// flat and deep: one field of 161×161×81 50.5 and 56.4 ms, 25 fields of 81×81×41 16.8 and 17.7, 10 of
// 161×161×81 72 and 101, 50 of 121×121×61 51 and 80, 24 of 401×401×121 678 and 1,130.)
const std::vector<TileShapeInfo>& tile_shapes() {
    static const std::vector<TileShapeInfo> shapes = {{0, kTileX, kTileY, kTileZ}};
    return shapes;
}

bool tile_known(int id) { return id >= 0 && id <= kTileLastId; }

namespace {

// A padded engine field → dense grid order, of another type with non-finite values as +inf, or of its own
// as it is. A warp per row.
template <typename From, typename To>
__global__ void dense_convert_kernel(const From* __restrict__ a, int pitch, int xoff, int nx, int64_t rows,
                                     To* __restrict__ b) {
    const int lane = threadIdx.x & 31;
    const int64_t nw = int64_t(gridDim.x) * (blockDim.x >> 5);
    for (int64_t r = (blockIdx.x * int64_t(blockDim.x) + threadIdx.x) >> 5; r < rows; r += nw) {
        const From* src = a + r * pitch + xoff;
        To* dst = b + r * nx;
        for (int q = lane; q < nx; q += 32) {
            const From v = src[q];
            if constexpr (std::is_same_v<From, To>) dst[q] = v;
            else dst[q] = finite_r(v) ? To(v) : To(__int_as_float(0x7f800000));
        }
    }
}

// One padded field on a grid to dense values of out_type at out (device), on s.
template <typename Real>
cudaError_t field_to_dense(const Real* T, const host::Grid& g, int pitch, int xoff, void* out, int out_type, cudaStream_t s) {
    const int64_t rows = int64_t(g.ny) * g.nz;
    const int blocks = int(std::min<int64_t>((rows + 7) / 8, 4096));
    if (out_type == TS_OUT_F64)
        dense_convert_kernel<Real, double><<<blocks, 256, 0, s>>>(T, pitch, xoff, g.nx, rows, static_cast<double*>(out));
    else
        dense_convert_kernel<Real, float><<<blocks, 256, 0, s>>>(T, pitch, xoff, g.nx, rows, static_cast<float*>(out));
    return cudaGetLastError();
}

}  // namespace

// Fields [f0, f1) of a job (after engine_run) in dense grid order of out_type, one after another at dst, on s.
template <typename Real>
static int fields_to_dense_device(ts_ctx* ctx, const EngineJob& job, size_t f0, size_t f1, void* dst, int out_type,
                                  cudaStream_t s) {
    char* d = static_cast<char*>(dst);
    const size_t osz = out_type == TS_OUT_F64 ? 8 : 4;
    for (size_t f = f0; f < f1; f++) {
        const host::Grid& g = *job.grids[job.fields[f].grid];
        TS_CUDA_TRY(ctx, field_to_dense(static_cast<const Real*>(job.fields[f].T), g, job.pitch[job.fields[f].grid],
                                        job.xoff, d, out_type, s));
        d += size_t(g.count()) * osz;
    }
    return TS_OK;
}

// Fields of the job to the host in dense grid order: made dense on the device in runs of fields, each run
// copied at once.
int fields_to_dense_host(ts_ctx* ctx, const EngineJob& job, int precision, void* out, int out_type) {
    const size_t osz = out_type == TS_OUT_F64 ? 8 : 4, most = size_t(512) << 20;
    char* dst = static_cast<char*>(out);
    for (size_t f0 = 0; f0 < job.fields.size();) {
        size_t f1 = f0, bytes = 0;
        while (f1 < job.fields.size()) {
            const size_t b = size_t(job.grids[job.fields[f1].grid]->count()) * osz;
            if (f1 > f0 && bytes + b > most) break;
            bytes += b;
            f1++;
        }
        void* stage = ctx->buf("out.stage", bytes);
        for (; !stage && f1 > f0 + 1; stage = ctx->buf("out.stage", bytes))  // no room: fewer fields at once
            bytes -= size_t(job.grids[job.fields[--f1].grid]->count()) * osz;
        if (!stage) return TS_E_NOMEM;
        int rc = precision == TS_PRECISION_F64
                     ? fields_to_dense_device<double>(ctx, job, f0, f1, stage, out_type, ctx->stream)
                     : fields_to_dense_device<Pair>(ctx, job, f0, f1, stage, out_type, ctx->stream);
        if (rc == TS_OK) rc = copy_to_host(ctx, dst, stage, bytes, ctx->stream);
        if (rc) return rc;
        dst += bytes;
        f0 = f1;
    }
    ctx->keep("out.stage");
    return TS_OK;
}

// One field as a dense float32 table on the device (the .qttb rounding).
int field_to_dense_f32_device(ts_ctx* ctx, const host::Grid& g, const FieldLayout& L, const void* T, int precision,
                              float* out, cudaStream_t s) {
    if (precision == TS_PRECISION_F64)
        TS_CUDA_TRY(ctx, field_to_dense(static_cast<const double*>(T), g, L.pitch, L.xoff, out, TS_OUT_F32, s));
    else
        TS_CUDA_TRY(ctx, field_to_dense(static_cast<const Pair*>(T), g, L.pitch, L.xoff, out, TS_OUT_F32, s));
    return TS_OK;
}

// Fields of a job as dense float32 tables on the device, one after another.
int fields_to_dense_f32_device(ts_ctx* ctx, const EngineJob& job, int precision, float* out) {
    for (const auto& f : job.fields) {
        const host::Grid& g = *job.grids[f.grid];
        FieldLayout L = field_layout(g, precision);
        int rc = field_to_dense_f32_device(ctx, g, L, f.T, precision, out, ctx->stream);
        if (rc) return rc;
        out += g.count();
    }
    return TS_OK;
}

FieldLayout field_layout(const host::Grid& g, int precision) {
    const int bx = kTileX, by = kTileY, bz = kTileZ;
    const int hx = 2;  // 16 bytes of 8-byte values (a double, or the FP32 precision's float pair)
    (void)precision;
    const int tx = (g.nx + bx - 1) / bx, ty = (g.ny + by - 1) / by, tz = (g.nz + bz - 1) / bz;
    FieldLayout L;
    L.pitch = hx + tx * bx + hx;
    L.xoff = hx;
    L.tiles = tx * ty * tz;
    L.mask_words = L.tiles * ((bx * by * bz + 31) / 32);
    L.rows_ = int64_t(g.ny) * g.nz;
    return L;
}

int64_t FieldLayout::elems() const { return int64_t(pitch) * rows_; }

static size_t up256(size_t b) { return (b + 255) / 256 * 256; }

int64_t FieldLayout::bytes(int precision) const {
    const size_t esz = 8;
    (void)precision;
    return int64_t(up256(size_t(elems()) * esz) + up256(size_t(tiles)) + up256(4 * size_t(mask_words)) + 256);
}

void engine_field_place(EngineField& f, const FieldLayout& L, int precision, void* block) {
    const size_t esz = 8;
    (void)precision;
    char* p = static_cast<char*>(block);
    f.T = p;
    p += up256(size_t(L.elems()) * esz);
    f.dirty = reinterpret_cast<uint8_t*>(p);
    p += up256(size_t(L.tiles));
    f.dmask = reinterpret_cast<uint32_t*>(p);
    p += up256(4 * size_t(L.mask_words));
    f.state = p;
}

template <typename Real>
int engine_run(ts_ctx* ctx, EngineJob& job, ts_eik_stats* stats) {
    if (job.fields.empty()) return TS_OK;
    const int precision = precision_of<Real>();
    const bool chosen = is_f64<Real>() ? ctx->chosen_f64 : ctx->chosen_f32;
    // Every field's buffers from one pooled block of the context.
    std::vector<FieldLayout> layouts;
    for (auto* g : job.grids) layouts.push_back(field_layout(*g, precision));
    size_t total = 0;
    for (auto& f : job.fields) total += size_t(layouts[f.grid].bytes(precision));
    char* pool = static_cast<char*>(ctx->buf("eng.fields", total));
    if (!pool) return TS_E_NOMEM;
    std::vector<EngineField*> fl;
    for (auto& f : job.fields) {
        engine_field_place(f, layouts[f.grid], precision, pool);
        pool += layouts[f.grid].bytes(precision);
        f.initialized = false;
        f.status = 0;
        fl.push_back(&f);
    }
    job.pitch.clear();
    for (auto& L : layouts) job.pitch.push_back(L.pitch);
    job.xoff = layouts.empty() ? 0 : layouts[0].xoff;
    // Small grids are solved in shared memory, a cluster per field, unless the caller has chosen the tiled
    // engine or wants the launch captured.
    ctx->resident_last = false;
    if (!chosen && !ctx->use_graph)
        if (const int cluster = resident_cluster(ctx, job))
            if (const auto rc = resident_run<Real>(ctx, job, cluster, stats, ctx->stream)) {
                ctx->resident_last = true;
                return *rc;
            }
    return engine_epoch<Real>(ctx, job.grids, job.metrics, fl, job.tol, job.wake_rel, 0, stats, ctx->stream);
}

template <typename Real>
int engine_run_to_host(ts_ctx* ctx, EngineJob& job, void* out, int out_type, ts_eik_stats* stats) {
    const size_t nf = job.fields.size(), half = (nf + 1) / 2;
    const size_t osz = out_type == TS_OUT_F64 ? 8 : 4;
    if (!ctx->copy_stream) TS_CUDA_TRY(ctx, cudaStreamCreateWithFlags(&ctx->copy_stream, cudaStreamNonBlocking));
    size_t bytes[2] = {0, 0};
    for (size_t f = 0; f < nf; f++) bytes[f < half ? 0 : 1] += size_t(job.grids[job.fields[f].grid]->count()) * osz;
    void* stage = ctx->buf("out.pipeline", std::max(bytes[0], bytes[1]));
    if (!stage) return TS_E_NOMEM;
    EventPair converted, copied;
    char* dst = static_cast<char*>(out);
    int rc = TS_OK;
    for (int part = 0; part < 2 && rc == TS_OK; part++) {
        const size_t f0 = part == 0 ? 0 : half, f1 = part == 0 ? half : nf;
        if (f0 == f1) continue;
        // The part as a job of its own (its fields move in and back out).
        EngineJob sub;
        sub.grids = job.grids;
        sub.metrics = job.metrics;
        sub.tol = job.tol;
        sub.wake_rel = job.wake_rel;
        for (size_t f = f0; f < f1; f++) sub.fields.push_back(std::move(job.fields[f]));
        rc = engine_run<Real>(ctx, sub, stats);
        if (rc == TS_OK) {
            // The stage is free once the previous part's copy has read it.
            if (part == 1) TS_CUDA_TRY(ctx, cudaStreamWaitEvent(ctx->stream, copied.a, 0));
            rc = fields_to_dense_device<Real>(ctx, sub, 0, sub.fields.size(), stage, out_type, ctx->stream);
        }
        if (rc == TS_OK) {
            TS_CUDA_TRY(ctx, cudaEventRecord(converted.a, ctx->stream));
            TS_CUDA_TRY(ctx, cudaStreamWaitEvent(ctx->copy_stream, converted.a, 0));
            TS_CUDA_TRY(ctx, cudaMemcpyAsync(dst, stage, bytes[part], cudaMemcpyDeviceToHost, ctx->copy_stream));
            TS_CUDA_TRY(ctx, cudaEventRecord(copied.a, ctx->copy_stream));
            dst += bytes[part];
        }
        job.pitch = sub.pitch;
        job.xoff = sub.xoff;
        for (size_t f = f0; f < f1; f++) job.fields[f] = std::move(sub.fields[f - f0]);
    }
    TS_CUDA_TRY(ctx, cudaStreamSynchronize(ctx->copy_stream));
    return rc;
}

template <typename Real>
int engine_run_in_parts(ts_ctx* ctx, EngineJob& job, void* out, int out_type, ts_eik_stats* stats) {
    const size_t nf = job.fields.size(), osz = out_type == TS_OUT_F64 ? 8 : 4;
    size_t per = (nf + 1) / 2;
    char* dst = static_cast<char*>(out);
    for (size_t f0 = 0; f0 < nf;) {
        const size_t f1 = std::min(nf, f0 + per);
        EngineJob sub;
        sub.grids = job.grids;
        sub.metrics = job.metrics;
        sub.tol = job.tol;
        sub.wake_rel = job.wake_rel;
        for (size_t f = f0; f < f1; f++) sub.fields.push_back(std::move(job.fields[f]));
        int rc = engine_run<Real>(ctx, sub, stats);
        bool settled = true;
        for (const auto& ef : sub.fields) settled = settled && ef.status == 1;
        if (rc == TS_OK && settled) rc = fields_to_dense_host(ctx, sub, precision_of<Real>(), dst, out_type);
        for (size_t f = f0; f < f1; f++) job.fields[f] = std::move(sub.fields[f - f0]);
        if (rc == TS_E_NOMEM && per > 1) {
            per = (per + 1) / 2;
            continue;
        }
        if (rc || !settled) return rc;  // the caller looks at the fields
        for (size_t f = f0; f < f1; f++) dst += size_t(job.grids[job.fields[f].grid]->count()) * osz;
        f0 = f1;
    }
    return TS_OK;
}

template int engine_run_in_parts<double>(ts_ctx*, EngineJob&, void*, int, ts_eik_stats*);
template int engine_run_in_parts<Pair>(ts_ctx*, EngineJob&, void*, int, ts_eik_stats*);
template int engine_run<Pair>(ts_ctx*, EngineJob&, ts_eik_stats*);
template int engine_run_to_host<double>(ts_ctx*, EngineJob&, void*, int, ts_eik_stats*);
template int engine_run_to_host<Pair>(ts_ctx*, EngineJob&, void*, int, ts_eik_stats*);
template int engine_run<double>(ts_ctx*, EngineJob&, ts_eik_stats*);

}  // namespace eik
}  // namespace ts
