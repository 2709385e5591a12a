// Copies between the caller's pageable memory and the device.
#pragma once

#include "ctx.h"
#include "ts_common.cuh"

namespace ts {

// bytes from device src, as stream s leaves it, to host dst; returns when dst holds them.
int copy_to_host(ts_ctx* ctx, void* dst, const void* src, size_t bytes, cudaStream_t s);

// The same for one of several copies: a copy that is not split over threads is only queued on s, and dst holds the
// bytes once s has been waited for.
int queue_to_host(ts_ctx* ctx, void* dst, const void* src, size_t bytes, cudaStream_t s);

// bytes from host src to device dst, after what stream s has queued; work queued on s afterwards sees
// them, and src may change when the call returns.
int copy_to_device(ts_ctx* ctx, void* dst, const void* src, size_t bytes, cudaStream_t s);

// Gives back what the copies of a context that is being destroyed used (its streams idle).
void free_copy_slots(ts_ctx* ctx);

// count doubles of the host as FP64 values, or as the FP32 precision's float pairs (formed on the device).
int upload_values(ts_ctx* ctx, double* dst, const double* src, size_t count, cudaStream_t s);
int upload_values(ts_ctx* ctx, Pair* dst, const double* src, size_t count, cudaStream_t s);

}  // namespace ts
