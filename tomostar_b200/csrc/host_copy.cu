// Copies between the caller's pageable memory and the device by several host threads.
//
// A cudaMemcpy to pageable memory is one host thread's copy through the driver's staging buffer, and
// into memory that has not been touched yet (what a caller has just allocated for a result) it is that
// thread's page faults: 200 MB took 92 ms (12 ms into memory already touched, 19 ms to the device), where
// the link itself takes 4. Here up to eight threads each move a part through two page-locked slots of
// their own, the device's copy of one slot running while the thread copies the other: 13 ms to the host
// and 7 ms to the device for the same 200 MB on a 16-core host.
#include <sys/mman.h>
#include <unistd.h>

#include <algorithm>
#include <atomic>
#include <cstring>
#include <thread>
#include <vector>

#include "host_copy.h"
#include "ts_common.cuh"

namespace ts {

namespace {

constexpr size_t kSlot = size_t(2) << 20;    // two per thread
constexpr size_t kSlotBytes = size_t(ts_ctx::kCopyStreams) * 2 * kSlot;
constexpr size_t kSmall = size_t(2) << 20;   // below this one plain copy is as fast
// Until another copy has made the streams, uploads below kFirst are plain copies as long as they have not added up to
// kAll: making the streams and locking the slots takes seven to ten ms once, a plain upload of 64 MB six, and a
// server that is given a few models never needs them. From then on a program's uploads gain: 400 rays on 21 MB of
// tables, call after call, 4.2 ms plain and 3.3 by threads.
constexpr size_t kFirst = size_t(64) << 20, kAll = 4 * kFirst;

// Runs part(k, slots) for k in [0, n) on n threads (this one among them; a thread that cannot be started
// leaves its part to this one). The first error of any part.
template <typename F>
cudaError_t on_threads(ts_ctx* ctx, int n, char* slots, F part) {
    std::atomic<int> err{int(cudaSuccess)};
    auto one = [&](int k) {
        cudaError_t e = cudaSetDevice(ctx->device);
        if (e == cudaSuccess) e = part(k, slots + size_t(k) * 2 * kSlot);
        int none = int(cudaSuccess);
        if (e != cudaSuccess) err.compare_exchange_strong(none, int(e));
    };
    std::vector<std::thread> pool;
    pool.reserve(size_t(n));
    for (int k = 1; k < n; k++) {
        try {
            pool.emplace_back(one, k);
        } catch (...) {
            one(k);
        }
    }
    one(0);
    for (auto& t : pool) t.join();
    return cudaError_t(err.load());
}

// Whether the pages of host memory are there (a sample of them): into memory touched before, one plain copy to
// the host is faster below 24 MB, where starting the threads takes longer than they save (2.5 MB 0.17 ms plain and
// 0.50 by threads, 8 MB 0.45 and 0.74, 24 MB 1.40 and 1.48, 32 MB 1.87 and 1.56); into new memory the threads
// share its page faults (2.5 MB 1.30 and 0.92, 8 MB 4.1 and 1.7).
constexpr size_t kTouched = size_t(24) << 20;
bool touched(const void* p, size_t bytes) {
    const size_t page = size_t(sysconf(_SC_PAGESIZE));
    for (int k = 0; k < 8; k++) {
        unsigned char there = 1;
        const uintptr_t at = (reinterpret_cast<uintptr_t>(p) + bytes / 8 * k) / page * page;
        if (mincore(reinterpret_cast<void*>(at), page, &there) == 0 && !(there & 1)) return false;
    }
    return true;
}

// The threads' page-locked slots, made on first use; null where they cannot be had. Locking 32 MB in huge pages
// takes 5 ms, touching them included; cudaHostAlloc took 15 to 17 for it.
char* page_locked_slots(ts_ctx* ctx) {
    if (ctx->copy_slots) return static_cast<char*>(ctx->copy_slots);
    void* p = mmap(nullptr, kSlotBytes, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
    if (p == MAP_FAILED) return nullptr;
    madvise(p, kSlotBytes, MADV_HUGEPAGE);  // (a wish: small pages do as well)
    std::memset(p, 0, kSlotBytes);
    if (cudaHostRegister(p, kSlotBytes, cudaHostRegisterDefault) != cudaSuccess) {
        cudaGetLastError();
        munmap(p, kSlotBytes);
        return nullptr;
    }
    ctx->copy_slots = p;
    return static_cast<char*>(p);
}

// Threads for a copy of this size, their streams and slots made on first use; 1: a plain copy.
int copy_threads(ts_ctx* ctx, const void* host, size_t bytes, bool to_host, char** slots) {
    if (bytes < kSmall) return 1;
    cudaPointerAttributes at{};
    const bool known = cudaPointerGetAttributes(&at, host) == cudaSuccess && at.type != cudaMemoryTypeUnregistered;
    cudaGetLastError();
    if (known) return 1;  // page-locked, managed or device memory: the driver's own copy, no host thread may touch it
    if (to_host && bytes < kTouched && touched(host, bytes)) return 1;
    if (!to_host && !ctx->copy_streams[0] && bytes < kFirst && (ctx->uploaded += bytes) < kAll) return 1;
    const unsigned cores = std::max(1u, std::thread::hardware_concurrency());
    const int n = int(std::min<size_t>({size_t(ts_ctx::kCopyStreams), size_t(std::max(1u, cores / 2)), bytes / (kSlot / 2)}));
    for (int k = 0; k < n; k++)
        if (!ctx->copy_streams[k] &&
            cudaStreamCreateWithFlags(&ctx->copy_streams[k], cudaStreamNonBlocking) != cudaSuccess) {
            cudaGetLastError();
            ctx->copy_streams[k] = nullptr;
            return 1;
        }
    *slots = page_locked_slots(ctx);
    return *slots ? n : 1;
}

struct SlotEvents {
    cudaEvent_t e[2] = {nullptr, nullptr};
    cudaError_t make() {
        for (auto& x : e) {
            const cudaError_t r = cudaEventCreateWithFlags(&x, cudaEventDisableTiming);
            if (r != cudaSuccess) return r;
        }
        return cudaSuccess;
    }
    ~SlotEvents() {
        for (auto& x : e)
            if (x) cudaEventDestroy(x);
    }
};

#define TS_STEP(call)                                \
    do {                                             \
        const cudaError_t r_ = (call);               \
        if (r_ != cudaSuccess) return r_;            \
    } while (0)

cudaError_t part_to_host(cudaStream_t s, char* dst, const char* src, size_t bytes, char* slots) {
    SlotEvents ev;
    TS_STEP(ev.make());
    auto fetch = [&](size_t o, int q) -> cudaError_t {
        TS_STEP(cudaMemcpyAsync(slots + q * kSlot, src + o, std::min(kSlot, bytes - o), cudaMemcpyDeviceToHost, s));
        return cudaEventRecord(ev.e[q], s);
    };
    if (bytes > 0) TS_STEP(fetch(0, 0));
    int q = 0;
    for (size_t o = 0; o < bytes; o += kSlot, q ^= 1) {
        if (o + kSlot < bytes) TS_STEP(fetch(o + kSlot, q ^ 1));
        TS_STEP(cudaEventSynchronize(ev.e[q]));
        std::memcpy(dst + o, slots + q * kSlot, std::min(kSlot, bytes - o));
    }
    return cudaSuccess;
}

cudaError_t part_to_device(cudaStream_t s, char* dst, const char* src, size_t bytes, char* slots) {
    SlotEvents ev;
    TS_STEP(ev.make());
    int q = 0;
    for (size_t o = 0; o < bytes; o += kSlot, q ^= 1) {
        const size_t n = std::min(kSlot, bytes - o);
        if (o >= 2 * kSlot) TS_STEP(cudaEventSynchronize(ev.e[q]));
        std::memcpy(slots + q * kSlot, src + o, n);
        TS_STEP(cudaMemcpyAsync(dst + o, slots + q * kSlot, n, cudaMemcpyHostToDevice, s));
        TS_STEP(cudaEventRecord(ev.e[q], s));
    }
    return cudaStreamSynchronize(s);
}

int copy(ts_ctx* ctx, void* dst, const void* src, size_t bytes, cudaStream_t s, bool to_host, bool wait = true) {
    if (bytes == 0) return TS_OK;
    char* slots = nullptr;
    const int n = copy_threads(ctx, to_host ? dst : src, bytes, to_host, &slots);
    if (n <= 1) {
        TS_CUDA_TRY(ctx, cudaMemcpyAsync(dst, src, bytes, to_host ? cudaMemcpyDeviceToHost : cudaMemcpyHostToDevice, s));
        if (wait) TS_CUDA_TRY(ctx, cudaStreamSynchronize(s));
        return TS_OK;
    }
    // The parts' streams follow what s has queued.
    struct After {
        cudaEvent_t e = nullptr;
        ~After() {
            if (e) cudaEventDestroy(e);
        }
    } after;
    TS_CUDA_TRY(ctx, cudaEventCreateWithFlags(&after.e, cudaEventDisableTiming));
    TS_CUDA_TRY(ctx, cudaEventRecord(after.e, s));
    for (int k = 0; k < n; k++) TS_CUDA_TRY(ctx, cudaStreamWaitEvent(ctx->copy_streams[k], after.e, 0));
    const size_t each = (bytes / size_t(n) + 4095) / 4096 * 4096;
    const cudaError_t e = on_threads(ctx, n, slots, [&](int k, char* mine) -> cudaError_t {
        const size_t b = std::min(bytes, each * size_t(k)), m = std::min(bytes, b + each) - b;
        char* d = static_cast<char*>(dst) + b;
        const char* f = static_cast<const char*>(src) + b;
        return to_host ? part_to_host(ctx->copy_streams[k], d, f, m, mine)
                       : part_to_device(ctx->copy_streams[k], d, f, m, mine);
    });
    if (e != cudaSuccess)  // no part may still be using the slots
        for (int k = 0; k < n; k++) cudaStreamSynchronize(ctx->copy_streams[k]);
    TS_CUDA_TRY(ctx, e);
    return TS_OK;
}

__global__ void pairs_kernel(const double* a, Pair* b, size_t n) {
    for (size_t q = blockIdx.x * size_t(blockDim.x) + threadIdx.x; q < n; q += size_t(gridDim.x) * blockDim.x)
        b[q] = Pair(a[q]);
}

}  // namespace

void free_copy_slots(ts_ctx* ctx) {
    if (!ctx->copy_slots) return;
    cudaHostUnregister(ctx->copy_slots);
    munmap(ctx->copy_slots, kSlotBytes);
    ctx->copy_slots = nullptr;
}

int copy_to_host(ts_ctx* ctx, void* dst, const void* src, size_t bytes, cudaStream_t s) {
    return copy(ctx, dst, src, bytes, s, true);
}

int queue_to_host(ts_ctx* ctx, void* dst, const void* src, size_t bytes, cudaStream_t s) {
    return copy(ctx, dst, src, bytes, s, true, false);
}

int copy_to_device(ts_ctx* ctx, void* dst, const void* src, size_t bytes, cudaStream_t s) {
    return copy(ctx, dst, src, bytes, s, false);
}

int upload_values(ts_ctx* ctx, double* dst, const double* src, size_t count, cudaStream_t s) {
    return copy_to_device(ctx, dst, src, count * sizeof(double), s);
}

int upload_values(ts_ctx* ctx, Pair* dst, const double* src, size_t count, cudaStream_t s) {
    // A pair has a double's size: the doubles go where the pairs will be and are replaced in place, each
    // by the thread that read it.
    static_assert(sizeof(Pair) == sizeof(double), "in place");
    if (count == 0) return TS_OK;
    if (int rc = copy_to_device(ctx, dst, src, count * sizeof(double), s)) return rc;
    pairs_kernel<<<int(std::min<size_t>((count + 255) / 256, 4096)), 256, 0, s>>>(reinterpret_cast<const double*>(dst),
                                                                                 dst, count);
    TS_CUDA_TRY(ctx, cudaGetLastError());
    return TS_OK;
}

}  // namespace ts
