// Fused batched RKF78 propagation kernels for sm_100a.
//
// One persistent kernel advances object groups through all their fixed steps:
// the RKF78 stages, the full force model and the 8th-order update run on
// chip (registers and shared memory), so the only per-object HBM traffic is the
// state read at the start and written at the end of the whole propagation.
//
// Work split (autotuned):  L lanes (1, 2, 4, 8 or 16) cooperate on one object,
// a warp holds 32/L objects.
//   * RK state: a lane of a group owns coordinate axes (position and velocity
//     in registers); the stage accelerations lie in shared memory, from which
//     the lane forms its axes' stage state (the reference's sums,
//     parm/integrate/rk/host/Step.h:33-104, with the position rows summed on
//     accelerations) and broadcasts it by warp shuffle.
//   * Spherical harmonics: the field's acceleration as column sums of solid
//     harmonics one degree up (geopotential.hpp), orders M in blocks of L
//     columns (2L where two lane groups share their columns: every lane then
//     runs its column for both groups' objects), from a lane-interleaved
//     coefficient tile that a TMA bulk copy stages into shared memory.  In
//     split precision the degrees above the FP64 low part run in FP32.  The
//     Earth's tide deltas (n <= 6) are summed apart, in FP64.  Partial
//     accelerations are folded across the group by xor shuffles.
//   * Everything else (third bodies, SRP with shadow, NRLMSISE-00 drag,
//     relativity) is evaluated by every lane of the group on the broadcast
//     stage state.
//
// Time grid: batches whose objects share epoch, step and duration read the
// per-step start / step size and the per-stage EpochRecord from tables made
// before the launch; mixed batches keep per-object time (FixedStep.h:30-37
// per object) and form each stage's record by 4-point Lagrange interpolation
// in an epoch-record grid of at most 30 s spacing that spans the batch, with
// the NRLMSISE-00 time inputs (seconds of day, sidereal time, weather slot)
// evaluated exactly at the stage epoch.
#pragma once
#include <stdint.h>

#include "device_env.cuh"
#include "geopotential.hpp"

namespace phop {

// Split precision keeps degrees n <= splitFp64Degree (by default 20, or 24
// for fields above degree 80; at most kLowMax) of every column in FP64, with
// a margin beyond (geopotential.hpp), and runs the rest in FP32.
constexpr int kLowDeg = 8;                                  // smallest FP64 low part of the split form
constexpr int kSplitFp64Degree = 20;                        // split form default up to degree 80
constexpr int kSplitFp64DegreeHigh = 24;                    // split form default above degree 80
constexpr int kLowMax = 24;                                 // largest FP64 low part

struct StepParams {
    DevEnv env;
    int64_t n;          // objects
    double* state;      // SoA: x[n], y[n], z[n], vx[n], vy[n], vz[n]
    const double* bc;   // cd * area / mass  (km^2 / kg)
    const double* ams;  // cr * area / mass
    // shared time grid
    int nsteps;
    const double* stepT0;
    const double* stepDt;
    const EpochRecord* records;  // [nsteps][13]
    // trajectory records (uniform batches): after every trajEvery-th step the
    // states go to traj[r][component][object], object in input order
    double* traj;
    int trajEvery;
    int trajRecords;  // capacity of traj in records: writes beyond it are skipped
    // per-object time (mixed batches)
    double* cur;
    const double* end;
    double* dt;
    const double* step;
    int64_t maxSteps;
    int* unfinished;        // per object: 1 if it did not reach its end
    const int64_t* order;   // processing order of objects (nullable)
    // epoch-record grid of a mixed batch (nullable): grid[k] holds the record
    // at TDB seconds (gridBase + k) * gridH, k < gridN.  The grid is anchored
    // at multiples of gridH, so an object's interpolated records do not depend
    // on which other objects share its batch.
    const EpochRecord* grid;
    // the same grid as value pairs: gridPairs[k * kInterpFields + f] = field f
    // of records k and k + 1, so that a 4-point stencil reads each field with
    // two 16-byte loads from two records instead of four 8-byte loads
    const double2* gridPairs;
    double gridH;
    int64_t gridBase;
    int gridN;
    int64_t stride;  // SoA stride of `state` (0: n); object pools use their capacity
    // geopotential
    const void* tile;       // tile entries in global memory
    int tileBytes;          // multiple of 16
    int nblocks;            // blocks of columns
    int lowDeg;             // split precision: FP64 low part
    const void* tile64;     // split precision: the FP64 tile (global memory) of L lanes
    int nblocks64;
    double splitRadius;     // split precision: radius (km) below which the tile part stays FP64; 0 = none
    int useSmemTile;
    int stagedBytes;        // of the tile in shared memory: all, or the first blocks (stepRoom)
    int streamTile;         // the tile streamed through rings in shared memory (hasStream shapes)
    int pairSh;             // the geopotential of lane-group pairs (tile built for 2L lanes)
    int duo;                // warps in pairs, the drag model on the second (hasDuo shapes)
    int nrl;                // the kernel with NRLMSISE-00 (a configuration that uses it needs it)
    int deepRegs;           // host-side choice of the kernel's thread bound (stepThreadBound)
    int tileWaitTest;       // test of the staging time-out: arm the barrier, issue no copy
    // scheduling and errors
    int* workCounter;
    int* errorFlag;
    int* tileFallbacks;     // CTAs whose tile staging timed out (read the tile from global memory); nullable
};

// shared memory of one object's stage accelerations: ten slots of three doubles
constexpr int kStageBytes = 10 * 3 * 8;

// Threads per CTA the step kernel is compiled for: narrow lane splits run one
// CTA of few threads per SM (the coefficient tile fills shared memory), so
// they get up to 255 registers per thread instead of spilling at 128.  The
// "wide" shape below, and at two and four lanes also a "deep" one of
// kDeepThreads threads: 255 registers a thread instead of 168 (fewer warps,
// fewer spills; the autotuner times both).
__host__ __device__ constexpr int maxStepThreads(int lanes) {
    return lanes == 1 ? 256 : lanes == 2 ? 320 : 384;
}
constexpr int kDeepThreads = 256;
__host__ __device__ constexpr bool hasDeepShape(int lanes) { return lanes == 2 || lanes == 4; }
// shapes that read shared memory by their own loads and can stream a tile
__host__ __device__ constexpr bool hasStream(int lanes, int deep) {
    return lanes == 1 || (deep && hasDeepShape(lanes));
}
// shapes that can hold the first blocks of a tile and read the rest from
// global memory
__host__ __device__ constexpr bool hasPart(int lanes, int deep) { return lanes >= 8 || (hasDeepShape(lanes) && !deep); }
// shapes with the drag model on a second warp, at the deep bound: two lane
// groups sharing columns up to four lanes, one object a lane at eight and
// sixteen
__host__ __device__ constexpr bool hasDuo(int lanes, int pair) { return lanes >= 8 ? !pair : pair != 0; }
__host__ __device__ constexpr int stepThreadBound(int lanes, int deep, int duo = 0) {
    return duo || (deep && hasDeepShape(lanes)) ? kDeepThreads : maxStepThreads(lanes);
}

// Shared memory of a step CTA: what a kernel holds by itself (the staging
// barrier; a duo kernel's mail, 7,296 bytes at one lane), the staged tile or
// the warps' rings, and the stage accelerations of the objects.  At least
// 1 KiB beside the dynamic part is left to the kernel.
constexpr int kDuoPairs = 4;  // warp pairs of a CTA of kDeepThreads threads
struct DuoMail {
    double f[3], sec, gast;
    int block, valid;
    double rho;
};
struct StepRoom {
    int threads = 0;          // most threads the shared memory has room for
    bool staged = false, streamed = false;  // the whole tile in shared memory; through rings there
    int stagedBytes = 0;      // whole tile, or its first blocks
};
// A tile that does not fit, or leaves room for fewer than three quarters of
// the threads, is streamed through a ring per warp where the kernel can (a
// streamed row costs about a fifth more than a staged one).  maxSmem: what a
// CTA may use in all; ownStaged, ownStreamed: what the kernels with and
// without a stream hold by themselves; bound: the threads asked for.  Where
// it neither fits nor streams (eight and sixteen lanes, the wide bound at two
// and four), its first blocks are staged beside the stage accelerations and
// the rest is read from global memory: with the rows of the solid harmonics a
// tile of eight or sixteen lanes fits to FP64 degree 84 or 80, with the former
// rows to 92 or 89, and read from global memory throughout, the field of one
// object at degree 88 took 3.4 ms for ten steps at its best shape; 2.08 with
// the former rows, 1.85 with the first blocks staged.
struct TileShape {
    int bytes, nblocks, W, degree, lowDeg;
};
inline StepRoom stepRoom(int maxSmem, int ownStaged, int ownStreamed, const TileShape& tile, int lanes, bool duo, int bound,
                         bool mayStage, bool mayStream, bool mayPart) {
    const int halves = duo ? 2 : 1;  // half of a duo CTA's warps hold objects
    const auto room = [&](int own) { return maxSmem - (own > 1024 ? own : 1024); };
    const auto fit = [&](int bytes) {
        return bytes < room(ownStaged) ? (room(ownStaged) - bytes) / kStageBytes * lanes / 32 * 32 * halves : 0;
    };
    const int staged = mayStage ? fit(tile.bytes) : 0;
    const int streamed = mayStream ? room(ownStreamed) / (kRingBytes + kStageBytes * (32 / lanes)) * 32 * halves : 0;
    const auto most = [&](int t) { return t < bound ? t : bound; };
    StepRoom r;
    r.streamed = mayStream && most(staged) < most(streamed) * 3 / 4;
    r.staged = !r.streamed && staged >= 64;
    r.threads = r.staged ? staged : r.streamed ? streamed : fit(0);
    if (r.staged) {
        r.stagedBytes = tile.bytes;
    } else if (mayStage && mayPart && !r.streamed) {
        r.stagedBytes = leadingBlocks(tile.nblocks, tile.W, tile.degree, tile.lowDeg,
                                      room(ownStaged) - kStageBytes * (most(r.threads) / halves / lanes));
    }
    return r;
}

void launchEpochRecords(const DevEnv& env, const double* epochs, int count, EpochRecord* out, cudaStream_t stream);
// pairs[(k * kInterpFields + f)] = {field f of grid[k], of grid[k + 1]}, k < count - 1
void launchRecordPairs(const EpochRecord* grid, int64_t count, double2* pairs, cudaStream_t stream);
cudaError_t launchPropagate(const StepParams& p, int lanes, bool split, bool shared, int ctas, int threads,
                            cudaStream_t stream);
int propagateSmemBytes(const StepParams& p, int lanes, int threads);
// 0 where the shape does not fit an SM
int propagateMaxCtasPerSm(int lanes, bool split, bool shared, int pair, int deep, int stream, int duo, int nrl, int threads, int smem);
// The compiled instantiation's attributes (maxThreadsPerBlock, numRegs,
// sharedSizeBytes): the launch shape never asks for more threads than the
// instantiation accepts, or more shared memory than its own leaves.
cudaError_t propagateAttributes(int lanes, bool split, bool shared, int pair, int deep, int stream, int duo, int nrl, cudaFuncAttributes* a);

}  // namespace phop
