// The resident solver's host interface: fields whose grid fits in the shared memory of one block
// cluster, solved there from the seeds to the settled field in one launch.
#pragma once

#include <optional>

#include "eik_engine.h"

namespace ts {
namespace eik {

// Blocks per cluster for this job, or 0 when some grid of it does not fit (the tiled engine's job).
int resident_cluster(ts_ctx* ctx, const EngineJob& job);

// Solves every field of the job to completion (the fields' buffers set as for engine_epoch; only the
// time array and the status and rounds are written). Nothing: the device does not take the launch, and no field
// has been touched (the tiled engine's job).
template <typename Real>
std::optional<int> resident_run(ts_ctx* ctx, EngineJob& job, int cluster, ts_eik_stats* stats, cudaStream_t s);

}  // namespace eik
}  // namespace ts
