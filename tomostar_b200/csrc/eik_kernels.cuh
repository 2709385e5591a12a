// Eikonal sweeping kernels: the plain per-plane kernel (the reference's launch scheme) and the
// tiled engine (one cooperative persistent launch over many fields and grids).
//
// Why the tiled engine gives the reference's result to the bit. A sweep of ordering `dir` visits
// the nodes by diagonal planes i'+j'+k' = p (mirrored coordinates), Gauss-Seidel in place
// (SphericalEikonal.cs:297-321). A node's update reads its neighbours one and two steps away on
// each axis; those on smaller p are already updated in this sweep, those on larger p are not yet.
// Any visiting order in which every node comes after its axis neighbours of smaller p produces
// exactly the same values. The engine cuts the grid into BX×BY×BZ tiles and visits a tile once the face
// neighbours before it along the sweep are done (the stencil only reaches face neighbours), and inside a
// tile goes by node planes. Every axis neighbour of smaller p lies in the same tile or in one of those,
// so the order is one of those orders; a tile's neighbours after it have finished the sweep before, so
// that sweeps may overlap.
// Skipping a tile none of whose nodes has an input that moved since its last evaluation skips
// only updates that would return the value already held, as the reference's dirty flags do
// (EikonalOpenCl.cs:529-532, 608-622); the field is unchanged by it.
#pragma once

#include "eik_update.cuh"

namespace ts {
namespace eik {

// ---- plain path: one launch per diagonal plane of one field (EikonalOpenCl.cs:232-268, 506-623) --

template <typename Real, bool VARZ>
__global__ void plain_sweep_kernel(Real* __restrict__ T, const Real* __restrict__ slow, const uint8_t* __restrict__ fixed,
                                   uint8_t* __restrict__ dirty, const Real* __restrict__ wx,
                                   const Real* __restrict__ wy, Real wz1, Real wz2, const Real* __restrict__ zc, int nx, int ny,
                                   int nz, int second, int* changed, int dir, int p, Real tol,
                                   unsigned long long* updates) {
    int i0 = max(0, p - (ny - 1) - (nz - 1));
    int iw = min(nx - 1, p) - i0 + 1;
    int k0 = max(0, p - (nx - 1) - (ny - 1));
    int a = blockIdx.x * blockDim.x + threadIdx.x;
    bool did = false;
    if (a < iw) {
        int ip = i0 + a, kp = k0 + int(blockIdx.y), jp = p - ip - kp;
        if (jp >= 0 && jp < ny) {
            int i = (dir & 1) ? nx - 1 - ip : ip;
            int j = (dir & 2) ? ny - 1 - jp : jp;
            int k = (dir & 4) ? nz - 1 - kp : kp;
            int nxy = nx * ny;
            int node = (k * ny + j) * nx + i;
            if (!fixed[node] && dirty[node]) {
                dirty[node] = 0;
                did = true;
                const Real inf = real_inf<Real>();
                Real cur = T[node];
                Real cand = Update<Real, VARZ>::eval(
                    slow[node], i > 0 ? T[node - 1] : inf, i + 1 < nx ? T[node + 1] : inf,
                    i > 1 ? T[node - 2] : inf, i + 2 < nx ? T[node + 2] : inf, j > 0 ? T[node - nx] : inf,
                    j + 1 < ny ? T[node + nx] : inf, j > 1 ? T[node - 2 * nx] : inf,
                    j + 2 < ny ? T[node + 2 * nx] : inf, k > 0 ? T[node - nxy] : inf,
                    k + 1 < nz ? T[node + nxy] : inf, k > 1 ? T[node - 2 * nxy] : inf,
                    k + 2 < nz ? T[node + 2 * nxy] : inf, wx[2 * (k * ny + j)], wx[2 * (k * ny + j) + 1],
                    wy[2 * k], wy[2 * k + 1], wz1, wz2, VARZ ? zc + kZCoef * k : nullptr, second != 0);
                if (cand < cur) {
                    T[node] = cand;
                    if (counts_as_change<Real>(cur, cand, tol)) atomicOr(changed, 1);
                    // Wake the nodes that read this one (EikonalOpenCl.cs:608-622).
                    if (i > 0) dirty[node - 1] = 1;
                    if (i > 1) dirty[node - 2] = 1;
                    if (i + 1 < nx) dirty[node + 1] = 1;
                    if (i + 2 < nx) dirty[node + 2] = 1;
                    if (j > 0) dirty[node - nx] = 1;
                    if (j > 1) dirty[node - 2 * nx] = 1;
                    if (j + 1 < ny) dirty[node + nx] = 1;
                    if (j + 2 < ny) dirty[node + 2 * nx] = 1;
                    if (k > 0) dirty[node - nxy] = 1;
                    if (k > 1) dirty[node - 2 * nxy] = 1;
                    if (k + 1 < nz) dirty[node + nxy] = 1;
                    if (k + 2 < nz) dirty[node + 2 * nxy] = 1;
                }
            }
        }
    }
    unsigned m = __ballot_sync(0xffffffffu, did);
    if ((threadIdx.x & 31) == 0 && m) atomicAdd(updates, (unsigned long long)__popc(m));
}

template <typename Real>
__global__ void fill_kernel(Real* __restrict__ p, Real v, int64_t n) {
    for (int64_t q = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; q < n; q += int64_t(gridDim.x) * blockDim.x) p[q] = v;
}

__global__ void fill_u8_kernel(uint8_t* __restrict__ p, uint8_t v, int64_t n);

// Writes seed times (already min-merged per field) and, for the plain path, the fixed mask.
template <typename Real>
__global__ void seed_kernel(Real* __restrict__ T, uint8_t* __restrict__ fixed, const int64_t* __restrict__ at,
                            const double* __restrict__ t, int count) {
    int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= count) return;
    T[at[q]] = Real(t[q]);
    if (fixed) fixed[at[q]] = 1;
}

// ---- tiled engine ---------------------------------------------------------------------------------

enum FieldStatus : int { kRunning = 0, kSettled = 1, kUnsettled = 2 };

// One grid shape and its metric (shared by every field solved on it).
struct GridDesc {
    int nx, ny, nz;
    int tx, ty, tz;            // tile counts
    int varz;                  // variable vertical spacing (extension)
    const void* wx;            // Real[2 * nz * ny]: longitude-axis weights (w1, w2) per (k, j)
    const void* wy;            // Real[2 * nz]: latitude-axis weights per k
    const void* zc;            // Real[kZCoef * nz] when varz
    double wz1, wz2;           // depth-axis weights of a uniform grid
    int pitch;                 // elements per padded field row (see FieldDesc::T)
};

// The engine's field layout: every (k, j) row is padded to `pitch` elements, node (i, j, k) at
// (k·ny + j)·pitch + HX + i with HX = 16 / sizeof(Real); the pads hold +inf and are never written.
// A tile's row segment with its two-node x halo is then one 16-byte-aligned run of whole chunks.
template <typename Real>
struct Layout {
    static constexpr int HX = 16 / int(sizeof(Real));
    TS_HDINL static int pitch(int tiles_x, int bx) { return HX + tiles_x * bx + HX; }
};

struct FieldState {
    int phase, round, status, changed;
    int rounds0, rounds1;
    // Tiles that have not finished the round in progress, and the rounds run in the current launch.
    int pending, launch_rounds;
};

template <typename Real>
struct FieldDesc {
    Real* T;              // the field, padded rows (Layout)
    const Real* s;        // its slowness
    uint8_t* dirty;       // one flag per tile: some node of the tile is due for an update
    uint32_t* dmask;      // per tile, one bit per node (MW words): the node is due for an update
    unsigned* tokens;     // per tile, what its next two sweeps have been given to start (flow scheduler)
    int seed_begin;       // its seed tiles: seed_tile[seed_begin .. seed_begin + seed_count), by tile id
    int seed_count;
    int cap;              // round cap per phase
    int seed_tile_lo, seed_tile_hi;  // smallest and largest seed tile id (no search outside)
    FieldState* state;               // the field's solve state; lives with the field between launches
    GridDesc g;                      // its grid (a copy: a visit's first loads do not wait for one another)
};

struct Control {
    int abort;
    int error;
    int running;
    int done;  // every field has stopped: the end of the launch
    unsigned long long updates;
    unsigned long long visits;
    // The tile queue's tickets: consumers take from head, producers reserve at tail.
    unsigned long long q_head, q_tail;
    unsigned long long t_start;  // globaltimer at the launch's start (first warp to arrive)
};

template <typename Real>
struct Args {
    const FieldDesc<Real>* fields;
    const int* seed_tile;        // tile id of each seed tile
    const uint32_t* seed_mask;   // kMaskWords words per seed tile: the fixed nodes
    Control* ctl;
    const volatile int* cancel;  // host-mapped cancel flag
    const int* field_list;       // the running fields
    int n_active;                // entries of field_list
    int max_rounds_per_launch;   // rounds this launch may run (<= 0: until every field is done)
    long long epoch_budget_ns;   // after this long, each field pauses at its next round end
    long long barrier_timeout_ns;
    // The tile queue, a bounded multi-producer multi-consumer ring of one word per slot: 0 while free, else a
    // tile (see TileItem) with the lap of its ticket. The producer of a ticket waits for its slot to be
    // free, its consumer for its lap; whoever takes a tile frees the slot.
    unsigned long long* q_slots;
    unsigned long long q_mask;
    int q_bits;                  // log2 of the slots
    Real tol;
    Real wake_rel;               // a drop wakes the neighbours when it exceeds wake_rel × the new time
    int causal;                  // a drop to t wakes only the neighbours holding more than t
};

TS_DEVINL unsigned long long global_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

}  // namespace eik
}  // namespace ts
