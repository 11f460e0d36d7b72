// staged.h — the staged path tracer (staged.cu): a path's ray casts and its
// shading in separate kernels, for every caller that renders whole samples of
// one scene (progressive passes, several passes at once, the batched
// renderer, the differentiable forward pass).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <mutex>
#include <vector>

#include "device_scene.h"

namespace zgl {

// Paths in flight at most: two states of float4 x 4 + uint2, a hit and a shadow
// ray each (200 B), 420 MB in all; a 1080p pass fits.
constexpr int64_t kStagedPaths = 1 << 21;
// Depth from which the one-kernel path tracer runs instead: the staged one
// launches two kernels per bounce whether or not a path gets there.
constexpr int32_t kStagedMaxDepth = 24;
// Sample indices whose Sobol rows fit the pool's table.
constexpr int32_t kStagedRows = 256;

// Order of the calls that share a pool: each waits on the device for the one
// before it, whatever streams they are enqueued on.
struct StagedTurns {
    std::mutex mutex;  // of one call's wait, launches and record
    cudaEvent_t done = nullptr;
    bool captured = false;       // a graph holds addresses of the pool
    std::vector<void*> retired;  // what such a graph may still use, freed with the pool
};

// Device memory of a staged render of up to `paths` paths at a time.
struct StagedPool {
    void* arena = nullptr;
    int64_t paths = 0;
    StagedTurns* turns = nullptr;  // from the first allocation on
    float4 *org[2], *dir[2], *thr[2], *pos[2];
    uint2* rng[2];
    int2* hit;
    float4 *sorg, *sdir, *scon;
    uint32_t* counts;  // per step: paths, shadow rays
    uint32_t* rows;    // kStagedRows x 256
};

// Pool for renders of `total` paths in place of what `p` holds; false without
// the memory (`p` is then as it was, and the caller keeps to one kernel or to
// the smaller pool).
bool staged_alloc(StagedPool& p, int64_t total);
void staged_free(StagedPool& p);
// Gives back memory that calls on the pool use beside it: at once, or with the
// pool if a graph may hold its address.
void staged_release(const StagedPool& p, void* memory);
// cudaMalloc of memory that the handle needs whether or not it runs staged:
// gives the pool back where there is not enough beside it.
cudaError_t staged_malloc_beside(StagedPool& p, void** memory, size_t bytes);

// Held while a call enqueues work on a pool (lists, counters, and whatever else
// of its handle such calls share).  Two calls that ran at once would append to
// the same lists, beyond their ends.  Captured calls take their turn when the
// graph runs: the wait and the record become nodes of it.
class StagedTurn {
public:
    StagedTurn(const StagedPool& pool, cudaStream_t st);
    ~StagedTurn();
    StagedTurn(const StagedTurn&) = delete;
    StagedTurn& operator=(const StagedTurn&) = delete;

private:
    StagedTurns* t_;
    cudaStream_t st_;
    bool captured_ = false;
    std::unique_lock<std::mutex> lock_;
};

// Samples s in [first, first + n) of every pixel of a scene, `maxDepth` at
// most kStagedMaxDepth.  Sample s uses Sobol row sample_offset(s) and
// freeCounter s + counter0; its radiance goes to out[(s - first) * npix +
// pix][3].  With `hits`, the first `castDepth` closest hits of each path go to
// hits[(k * n + s - first) * npix + pix] and the occlusion answers of its
// first 32 light samples to vis[(s - first) * npix + pix].
struct StagedJob {
    DeviceScene sc;
    int32_t maxDepth, rr, rrStart, sampleLight, uniformSel;
    float portion;
    bool full;  // metal-workflow or dielectric materials
    int32_t first, n, counter0;
    float* out;
    int2* hits;
    int32_t castDepth;
    uint32_t* vis;
};
cudaError_t launch_staged(const StagedPool& pool, const StagedJob& job, cudaStream_t st);

// Light paths [0, paths) of one pass, path k with randSeed seed + k, splatted
// into `film` (RGB floats).  `triple`: the triple integrator's light half, its
// connections scaled by `scale`.  `maxDepth` at most kStagedMaxDepth.
struct StagedLightJob {
    DeviceScene sc;
    int32_t maxDepth, rr, rrStart;
    bool full, triple;
    uint32_t paths, seed;
    float scale;
    float* film;
};
cudaError_t launch_staged_light(const StagedPool& pool, const StagedLightJob& job, cudaStream_t st);

// Sobol rows of samples [row0, row0 + n), n at most kStagedRows, into the pool.
cudaError_t launch_staged_rows(const StagedPool& pool, const uint32_t* mats, int32_t row0, int32_t n,
                               cudaStream_t st);
// SMs of the current device.
int staged_sms();

// Whether a scene and depth run staged.
inline bool staged_covers(const DeviceScene& sc, int32_t maxDepth) {
    return sc.accel.wide != nullptr && maxDepth >= 0 && maxDepth <= kStagedMaxDepth;
}
// Whether it is the faster way for a call of `paths` paths, in one pass or
// several.  Two launches a bounce have a latency (about 65 us at depth 5) that
// few paths do not fill, all the less where many of them miss the scene.  One
// pass of a small scene, time of one kernel over staged, square film at depth
// 3, at 7, and film three times as wide as high (which sees past the box) at
// depth 3: 2k triangles 60k paths 0.93, 1.03, 0.83, 100k 1.04, 1.27, 0.83,
// 130k 1.15, 1.40, 0.91, 160k 1.17, 1.40, 1.00; all material types 60k 1.13,
// 1.46, 0.86, 100k 1.40, 2.07, 0.95, 130k 1.55, 2.20, 1.08.  100k triangles,
// us, 16k paths 456 and 507, 32k 650 and 558.  The kernel of several passes
// has 32 registers: 8k paths 1.14-1.22 times the staged time, 20k 1.03-1.12,
// 90k 1.00-1.52.
inline bool staged_pays(const DeviceScene& sc, int64_t paths, bool several, bool full) {
    if (several) return paths >= 8192;
    if (sc.accel.M >= 16384) return paths >= 32768;
    return paths >= (full ? 131072 : 147456);
}
// A differentiable step, forward and replay (2k triangles, depth 6, us): 16k
// paths 702 in one kernel each and 709 staged, 33k 789 and 767, 65k 1043 and
// 842.
inline bool staged_diff_pays(int64_t paths) { return paths >= 32768; }
// Whether a request of a batch leaves the launch it shares with the others:
// what fills the GPU there is the others' paths too.
inline bool staged_pays_in_batch(const DeviceScene& sc, int64_t paths) {
    return paths >= 98304 || (sc.accel.M >= 16384 && paths >= 32768);
}
// The same for light paths (depth 8; one kernel, staged): 49k on 20k triangles
// 0.55, 0.61 ms, on 200k 1.78, 1.03; 98k on 2k triangles 0.76, 0.57.
inline bool staged_light_pays(const DeviceScene& sc, int64_t paths) {
    return paths >= 98304 || (sc.accel.M >= 131072 && paths >= 32768);
}
// Paths of n samples per pixel, film edges padded to whole tiles.
inline int64_t staged_paths(int32_t filmW, int32_t filmH, int64_t n) {
    return (int64_t)((filmW + 7) / 8) * ((filmH + 3) / 4) * 32 * n;
}

}  // namespace zgl
